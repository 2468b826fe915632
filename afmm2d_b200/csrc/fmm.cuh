// Tree views handed to the sweep kernels (see fmm.cu, mixed.cu).
#pragma once
#include <stdint.h>

#include <algorithm>
#include <string>
#include <vector>

#include "afmm_internal.cuh"

namespace afmm {

constexpr int kMaxLevels = 16;

// The split of the SM's memory between shared memory and L1 that the kernels of
// one product ask for (about 100 KB shared): an SM changes it only when it is
// empty, so kernels that differ in it do not run side by side on one SM.
// (300,000 points, mixed: 530 -> 448 us; 28%, 58%, 100%: 512, 482, 528.)
constexpr int kCarveoutPercent = 44;
template <class F>
inline void same_carveout(F* fn) {
  AFMM_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, kCarveoutPercent));
}

// Launch on stream s, with `early` as a programmatic dependent of the kernel before it: its
// CTAs may start (tables, operators into L2) as soon as all of that kernel's
// have, and wait at dep_wait() for its end.  The product's chain of small
// kernels (a level is a launch) then loses neither the launch gap nor the
// latency of the tables: 4,096 points, one column, 57 -> 50 us; 100,003 points
// 265 -> 225 us.
template <class... P, class... A>
inline void launch_dependent(bool early, void (*fn)(P...), long grid, int block, size_t smem, cudaStream_t s,
                             A&&... args) {
  same_carveout(fn);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  AFMM_CUDA(cudaLaunchKernelEx(&cfg, fn, static_cast<P>(args)...));
}
// Lets the next dependent launch start once every CTA has got here.
__device__ __forceinline__ void dep_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Waits for the end of the kernel that this one depends on (none: returns at
// once); only constant data is read before.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Device pointers of one level, passed by value to kernels.
struct LevelView {
  long nbox = 0;
  const int32_t* il = nullptr;
  const int32_t* rank = nullptr;
  const int32_t* skel_off = nullptr;
  const int32_t* node_off = nullptr;
  const int32_t* leaf_start = nullptr;  // leaf level only (quadtree order)
  const int64_t* l2p_off = nullptr;
  const double* l2p = nullptr;     // column-major (row index fastest)
  const double* l2p_rm = nullptr;  // row-major copy (rank index fastest)
  const int64_t* m2l_off = nullptr;
  long box0 = 0, nrun = 0;  // boxes of the one-column L2L (a shard's, else all)
  double* m2l = nullptr;
  const double2* skel_xy = nullptr;
  double* qhat = nullptr;
  double* yhat = nullptr;
  const int32_t* skel_box = nullptr;  // skeleton row -> box
  const int32_t* grp_box = nullptr;   // row group (<= 8 rows of one box) -> box
  const int32_t* grp_row = nullptr;   // row group -> first skeleton row
  long ngroups = 0;
  const int32_t* cgrp_box = nullptr;  // row chunk (<= kChunkRows rows of one box) -> box
  const int32_t* cgrp_row = nullptr;  // row chunk -> first skeleton row
  long ncgroups = 0;
  const int32_t* ncgrp_box = nullptr;  // node-row chunk (<= kChunkRows node rows of one box) -> box
  const int32_t* ncgrp_row = nullptr;  // node-row chunk -> first node row
  long nncgroups = 0;
  const int32_t* ptile_par = nullptr;  // parent row tile (<= 128 rows of 4 children) -> parent box
  const int32_t* ptile_row = nullptr;  // parent row tile -> first row of the children's concatenated rows
  long nptiles = 0;
  const int32_t* tile_box = nullptr;  // row tile (<= 128 skeleton rows of one box) -> box
  const int32_t* tile_row = nullptr;  // row tile -> first row within the box (a multiple of 8)
  long ntiles = 0;
  unsigned char* m2l_s = nullptr;      // byte-plane blocks (m2l_i8_k.cuh; null when not stored)
  const int64_t* m2l_s_off = nullptr;
  unsigned char* qs8 = nullptr;        // charges' byte planes of the current pass
  const int32_t* qs8_off = nullptr;
  int32_t* qs_exp = nullptr;
  int64_t* qs_sum = nullptr;
  uint32_t* m2l_q = nullptr;          // 32-bit fixed-point blocks (null when not stored)
  double2* m2l_dec = nullptr;         // per (box, slot) decode constants
  // one-column M2L (m2l_pair_box): per box its forward columns, the columns'
  // sums (box b's from back_off[b] on) and where a box finds its own among
  // them (kForwardSlots per box, -1 = none); the boxes to run for a shard
  // (null: all)
  struct ForwardBox* fwd = nullptr;
  double* back = nullptr;
  const int64_t* back_off = nullptr;
  int64_t* back_src = nullptr;
  const int32_t* m2l_run = nullptr;
  long nm2l_run = 0;
  long nrows = 0;                     // skeleton rows (sum of ranks)
  long nnodes = 0;                    // node rows (sum of node counts)
};

// Levels 2..L and the prefix of their skeleton row counts: the M2L kernels
// run one thread per skeleton row over this flat row space.
struct LevelSet {
  int nlev = 0;
  LevelView lv[kMaxLevels];
  long row0[kMaxLevels + 1] = {0};
  long grp0[kMaxLevels + 1] = {0};   // prefix of row-group counts
  long cgrp0[kMaxLevels + 1] = {0};  // prefix of row-chunk counts
  long pt0[kMaxLevels + 1] = {0};    // prefix of parent row-tile counts
  long t0[kMaxLevels + 1] = {0};     // prefix of 128-row tile counts
  long b0[kMaxLevels + 1] = {0};     // prefix of box counts
  long m0[kMaxLevels + 1] = {0};     // prefix of the boxes that the one-column M2L runs (a shard's, else all)
  int src[kMaxLevels] = {0};         // index of entry j among levels 2..L (per-level device tables)
  uint32_t pf_ahead = 12 * 1024;     // L2 prefetch window of the stored-block M2L kernels (bytes)
};

// The levels of `ls` whose bit in `mask` (bit t = entry t) equals `keep`,
// with their prefixes rebuilt and their original indices kept in src.
inline LevelSet level_subset(const LevelSet& ls, uint32_t mask, bool keep) {
  LevelSet o;
  o.pf_ahead = ls.pf_ahead;
  for (int t = 0; t < ls.nlev; ++t) {
    if ((((mask >> t) & 1u) != 0) != keep) continue;
    const int n = o.nlev;
    o.lv[n] = ls.lv[t];
    o.src[n] = ls.src[t];
    o.row0[n + 1] = o.row0[n] + (ls.row0[t + 1] - ls.row0[t]);
    o.grp0[n + 1] = o.grp0[n] + (ls.grp0[t + 1] - ls.grp0[t]);
    o.cgrp0[n + 1] = o.cgrp0[n] + (ls.cgrp0[t + 1] - ls.cgrp0[t]);
    o.pt0[n + 1] = o.pt0[n] + (ls.pt0[t + 1] - ls.pt0[t]);
    o.t0[n + 1] = o.t0[n] + (ls.t0[t + 1] - ls.t0[t]);
    o.b0[n + 1] = o.b0[n] + (ls.b0[t + 1] - ls.b0[t]);
    o.m0[n + 1] = o.m0[n] + (ls.m0[t + 1] - ls.m0[t]);
    ++o.nlev;
  }
  return o;
}

// Tunable launch parameters of a handle (afmm_autotune / afmm_set_tuning);
// none of them changes the FP64 path's arithmetic.
struct Tuning {
  uint32_t pf_fp64 = 12 * 1024;     // L2 prefetch window of the one-column FP64 / mixed M2L (bytes)
  uint32_t pf_batched = 12 * 1024;  // L2 prefetch window of the batched stored-block M2L (bytes)
  uint32_t otf_mixed = 0;           // bit t: level t + 2 evaluated on the fly in the one-column mixed path
  uint32_t otf_batched = 0;         // bit t: level t + 2 evaluated on the fly in batched mixed passes
  int host_pass_cols = 0;           // columns per pass of host-pointer batched calls (0: automatic)
  int m2l_t16 = 0;                  // 16-column stored M2L on transposed m16n8k4 tiles (else 8x8x4 tiles)
  int p2p_tc = 0;                   // 16-column mixed near field on tcgen05 tiles (else mma.sync tiles)
  int m2l_tc = 0;  // 16-column mixed stored M2L on tcgen05: 2 exact integer products from the byte
                   // planes; 1 TF32 tiles, an FP32 far field outside the mixed tolerance on deep trees,
                   // never chosen by the autotuner; 0 FP64 tiles
};

// Grid cell (ix, iy) of box k at level j: the base-4 digits of k read as
// child offsets 0:(0,0) 1:(1,0) 2:(1,1) 3:(0,1) (src/AFMM2DTree.cpp:978-986),
// and the inverse.
__device__ __forceinline__ void cell_of(long k, int j, int& ix, int& iy) {
  int x = 0, y = 0;
  for (int l = j - 1; l >= 0; --l) {
    int d = (int)((k >> (2 * l)) & 3);
    x = 2 * x + (d == 1 || d == 2);
    y = 2 * y + (d >= 2);
  }
  ix = x;
  iy = y;
}

__device__ __forceinline__ long box_of(int ix, int iy, int j) {
  long k = 0;
  for (int l = j - 1; l >= 0; --l) {
    int bx = (ix >> l) & 1, by = (iy >> l) & 1;
    k = 4 * k + (by ? (bx ? 2 : 3) : (bx ? 1 : 0));
  }
  return k;
}

// L2 prefetch of a global range: cp.async.bulk.prefetch.L2 (16-byte aligned
// start, size a multiple of 16).  Issued by one lane.
__device__ __forceinline__ void prefetch_l2_bulk(uintptr_t p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Streams a box's contiguous M2L region into L2 ahead of the warp that
// consumes it in order: `advance(pos)` keeps the prefetched front `ahead`
// bytes beyond `pos` (0: no prefetch), in kStep pieces (the last piece may
// extend < 16 bytes past the region; the block allocations are padded for
// that).
struct L2Stream {
  static constexpr uintptr_t kStep = 4096;
  uintptr_t front, end, ahead;
  __device__ __forceinline__ L2Stream(const void* begin, const void* stop, uintptr_t window)
      : front((uintptr_t)begin & ~(uintptr_t)15), end((uintptr_t)stop), ahead(window) {}
  __device__ __forceinline__ void advance(const void* pos, int lane) {
    uintptr_t upto = (uintptr_t)pos + ahead;
    if (upto > end) upto = end;
    while (front < upto) {  // warp-uniform
      if (lane == 0) {
        const uintptr_t left = (end - front + 15) & ~(uintptr_t)15;
        prefetch_l2_bulk(front, (uint32_t)(left < kStep ? left : kStep));
      }
      front += kStep;
    }
  }
};

// Prefetches [begin, end) into L2 in 4 KB pieces spread over the warp's
// lanes (start rounded down to 16 bytes, end up to 16 bytes: the arrays are
// allocated with that much padding).
__device__ __forceinline__ void prefetch_l2_region(const void* begin, const void* end, int lane) {
  const uintptr_t a = (uintptr_t)begin & ~(uintptr_t)15;
  const uintptr_t e = ((uintptr_t)end + 15) & ~(uintptr_t)15;
  for (uintptr_t p = a + (uintptr_t)lane * 4096; p < e; p += 32 * 4096) {
    const uintptr_t left = e - p;
    prefetch_l2_bulk(p, (uint32_t)(left < 4096 ? left : 4096));
  }
}

// Value of a 32-bit fixed-point M2L entry: the double with high word
// 0x43300000 and low word u is 2^52 + u exactly, so one FMA with the block's
// decode constants (2^k, -(2^52 + 2^31) 2^k) gives (u - 2^31) 2^k exactly.
__device__ __forceinline__ double decode_q32(uint32_t u, double2 dec) {
  return fma(__hiloint2double(0x43300000, (int)u), dec.x, dec.y);
}

// Leaf-level data for the near field.
struct NearView {
  long nleaf = 0;  // leaves of the launch: leaf0 .. leaf0 + nleaf - 1 (a shard's range, else all)
  long leaf0 = 0;
  int nmax = 0;
  const double2* pts = nullptr;        // sorted points
  const int32_t* leaf_start = nullptr; // quadtree order
  const int32_t* leaf_cnt = nullptr;
  const int32_t* nbr = nullptr;        // nleaf * 8
  const double2* anchor = nullptr;     // leaf anchors (FP64)
  const float2* rel = nullptr;         // point minus its leaf anchor (FP32), sorted order
  const float* span = nullptr;         // per leaf max |rel| component
  // FP64 near field of one column (near_leaf): its outputs, and for a shard
  // the leaves to run (the shard's own, and those that hold a pair with one of
  // its leaves); null: leaves leaf0 .. leaf0 + nleaf - 1
  double* part = nullptr;  // kNearParts x n
  long n = 0;              // points
  const int32_t* run = nullptr;
  long nrun = 0;
};
// Near-field sums of a point: its leaf's own work, and what the four leaves
// before it (neighbour slots 4..7) worked out for it.
constexpr int kNearParts = 5;

// CUDA-event marks for per-stage device timing.
struct StageTimer {
  std::vector<std::pair<std::string, cudaEvent_t>> marks;
  size_t used = 0;
  // stages run one after another on the launching stream (no near field
  // beside the far field), so every stage is its kernels' own duration
  bool serial = false;
  // spans timed on another stream (a stage that overlaps the marked ones)
  struct Span {
    std::string name;
    cudaEvent_t b, e;
  };
  std::vector<Span> spans;
  size_t nspans = 0;
  void reset() {
    used = 0;
    nspans = 0;
  }
  int span_begin(cudaStream_t s, const char* name) {
    if (nspans == spans.size()) {
      Span sp{name, nullptr, nullptr};
      cudaEventCreate(&sp.b);
      cudaEventCreate(&sp.e);
      spans.push_back(sp);
    }
    spans[nspans].name = name;
    cudaEventRecord(spans[nspans].b, s);
    return (int)nspans++;
  }
  void span_end(cudaStream_t s, int i) { cudaEventRecord(spans[(size_t)i].e, s); }
  void mark(cudaStream_t s, const char* name) {
    if (used == marks.size()) {
      cudaEvent_t e;
      cudaEventCreate(&e);
      marks.push_back({name, e});
    }
    marks[used].first = name;
    cudaEventRecord(marks[used].second, s);
    ++used;
  }
  // durations between consecutive marks, accumulated by name
  void collect(std::vector<std::pair<std::string, double>>& out) {
    out.clear();
    for (size_t i = 0; i + 1 < used; ++i) {
      float ms = 0;
      cudaEventElapsedTime(&ms, marks[i].second, marks[i + 1].second);
      bool found = false;
      for (auto& o : out)
        if (o.first == marks[i].first) {
          o.second += ms;
          found = true;
        }
      if (!found) out.push_back({marks[i].first, ms});
    }
    for (size_t i = 0; i < nspans; ++i) {
      float ms = 0;
      cudaEventElapsedTime(&ms, spans[i].b, spans[i].e);
      bool found = false;
      for (auto& o : out)
        if (o.first == spans[i].name) {
          o.second += ms;
          found = true;
        }
      if (!found) out.push_back({spans[i].name, ms});
    }
  }
  ~StageTimer() {
    for (auto& m : marks) cudaEventDestroy(m.second);
    for (auto& sp : spans) {
      cudaEventDestroy(sp.b);
      cudaEventDestroy(sp.e);
    }
  }
};

constexpr int kSmallProduct = 1 << 19;  // points
struct MatvecPlan {
  int N = 0, L = 0;
  KernelParams kp;
  const int64_t* perm = nullptr;
  const int32_t* iperm = nullptr;  // original index -> sorted position
  double* qs = nullptr;  // sorted charges
  double* ys = nullptr;  // sorted potentials
  LevelView lv[kMaxLevels];
  int rmax[kMaxLevels] = {0};   // largest rank per level
  int n1max[kMaxLevels] = {0};  // largest node count per level
  LevelSet levels;       // levels 2..L for the M2L launch
  NearView near;
  // the near field of a one-column product runs beside the far field, into
  // near.part, one of them on a stream of lower / higher priority than the
  // product's own (beside_near); the scatter adds the two
  cudaStream_t s_near = nullptr, s_far = nullptr;
  cudaEvent_t ev_q = nullptr, ev_side = nullptr;
  bool small() const { return N < kSmallProduct; }
  Tuning tune;
  // A shard of one problem (afmm_set_shard): the stored-block M2L and the
  // L2L of the levels at and below shard_level, and the near field, run only
  // over the shard's subtrees (contiguous box ranges); the gather, the M2M,
  // the on-the-fly M2L and the upper levels run whole on every shard, and the
  // potentials of points outside the shard come out as zeros.  Unsharded,
  // these equal levels / lv / near.
  int shard_index = 0, shard_count = 1, shard_level = 0;
  LevelSet levels_m2l;
  LevelView lv_down[kMaxLevels];
  NearView near_own;
};

// The near and the far field of a one-column product, after what is queued on s
// so far and before what follows: near(stream), far(stream).  Below
// kSmallProduct points the far field's chain of small kernels is the longer
// path: it follows on s at once, as dependent launches, and the near field
// goes to the side.  Above, the near field follows on s and fills the GPU
// first, and the far field takes slots as the near field's CTAs leave them (its
// stream has the higher priority): it so runs in the near field's tail too,
// where large leaves leave most SMs idle.  Time of the second way over the first,
// FP64 / mixed, over leaves of 32 to 391 points and four kernels: 0.89-1.13 /
// 0.96-1.18 up to 131,072 points (above 1 with leaves of 32 to 64: there the chain is
// the longer path, and two streams' launches cost 10 us), 0.96-1.05 / 0.94-1.13 at
// 262,144, 0.85-1.02 / 0.93-1.01 at 400,000, 0.86-1.02 / 0.90-1.02 at 600,000 and more
// (1,048,576 points, mixture, 1/r 1.29 -> 1.12 ms; uniform, log, leaves of 256 3.41 ->
// 3.48).  The line is where nothing loses more than 2% any longer.
template <class Near, class Far>
inline void beside_near(const MatvecPlan& p, cudaStream_t s, StageTimer* tm, Near&& near, Far&& far) {
  if (tm && tm->serial) {
    far(s);
    if (tm) tm->mark(s, "p2p");
    near(s);
    return;
  }
  const cudaStream_t sn = p.small() ? p.s_near : s, sf = p.small() ? s : p.s_far;
  AFMM_CUDA(cudaEventRecord(p.ev_q, s));
  AFMM_CUDA(cudaStreamWaitEvent(p.small() ? sn : sf, p.ev_q, 0));
  const int sp = tm ? tm->span_begin(sn, "p2p_kernel") : -1;  // the kernel's own duration
  near(sn);
  if (tm) tm->span_end(sn, sp);
  if (p.small()) AFMM_CUDA(cudaEventRecord(p.ev_side, sn));
  far(sf);
  if (tm) tm->mark(sf, "p2p");  // (the "p2p" stage is the wait for the near field)
  if (!p.small()) AFMM_CUDA(cudaEventRecord(p.ev_side, sf));
  AFMM_CUDA(cudaStreamWaitEvent(s, p.ev_side, 0));
}

// Level and box range [k0, k1) of shard `index` of `count` on a tree of
// levels 2..L: the shallowest level with at least four boxes per shard (the
// deepest level when none has), boxes split evenly (a KD tree's boxes of one
// level hold equal point counts).  Returns false when the tree has fewer
// leaves than shards.
inline bool shard_range(int L, int index, int count, int& level, long& k0, long& k1) {
  if (count < 1 || index < 0 || index >= count || L < 2) return false;
  level = L;
  for (int j = 2; j <= L; ++j)
    if ((1L << (2 * j)) >= 4L * count) {
      level = j;
      break;
    }
  const long nb = 1L << (2 * level);
  if (nb < count) return false;
  k0 = nb * index / count;
  k1 = nb * (index + 1) / count;
  return true;
}

// Warps per CTA of the FP64 near field of leaves of up to nmax points
// (near_leaf): the leaf's five source leaves make blocks of 32 points, up to
// kNearJ of them a warp at a time.
constexpr int kNearJ = 2;
inline int near_warps(int nmax) {
  const int blocks = (5 * nmax + 31) / 32;
  int best = 1;
  double fill = 0.0;  // how evenly the warps share the blocks
  for (int w = 1; w <= 8; ++w) {
    const int per = (blocks + w - 1) / w;  // blocks of the busiest warp
    const double f = (double)blocks / (per * w) - (per > 2 * kNearJ && w < 8 ? 1.0 : 0.0);
    if (f >= fill) {
      fill = f;
      best = w;
    }
  }
  return best;
}
// A warp goes round the n targets, lane l from target l on; with fewer than 32
// the lanes go round in groups of n, each group with target sums of its own.
// The targets are repeated behind their end, and a row of target sums is as
// long, so that no lane's index wraps.
__host__ __device__ __forceinline__ int near_row(int n) { return n >= 32 ? n + 32 : 2 * n * ((31 + n) / n); }
constexpr int kNearRowMax = 128;  // of n < 32
inline size_t near_smem(int nmax, int warps) {
  const size_t row = std::max(near_row(nmax), kNearRowMax);
  return row * (sizeof(double2) + sizeof(double)) + nmax * sizeof(double) + (size_t)warps * row * sizeof(double);
}
// ------------------------------------------------ FP64 sweep rows
// The arithmetic of one output of each FP64 sweep, shared by the
// single-problem kernels (fmm.cu) and the fused many-problem kernels (set.cu)
// so both give the same bits.

// Loads of values that may have been written earlier in the same launch (the
// persistent many-problem sweeps): kL2 reads them through L2 (ld.global.cg),
// which other SMs' published stores reach; otherwise an ordinary load.
template <bool kL2>
__device__ __forceinline__ double ld_src(const double* p) {
  if constexpr (kL2) return __ldcg(p);
  else return *p;
}

// y += A x for the rows of one panel (NT tiles of 8 rows, nrow of them) by one
// warp: A column-major with leading dimension lda, at the panel's first row.
// Lane (rsub, csub) holds rows 8 k + rsub of columns 4 j + csub; up to 40 loads
// per lane are independent, so a box's operator is asked for in one go.
// Afterwards every lane holds its rows' sums.
template <int NT, bool FULL, bool kL2>
__device__ __forceinline__ void gemv_group(const double* __restrict__ P, long lda, int left, bool last,
                                           const double* x, double (&y)[NT]) {
  const int csub = (threadIdx.x & 31) >> 3;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const bool vc = FULL || 4 * j + csub < left;
    const double xv = vc ? ld_src<kL2>(x + 4 * j) : 0.0;
#pragma unroll
    for (int k = 0; k < NT; ++k) {
      const double m = vc && (k + 1 < NT || last) ? __ldg(P + 4 * j * lda + 8 * k) : 0.0;
      y[k] += m * xv;
    }
  }
}
template <int NT, bool kL2>
__device__ __forceinline__ void gemv_panel(const double* __restrict__ A, long lda, int nrow, int cols,
                                           const double* x, double (&y)[NT]) {
  const int lane = threadIdx.x & 31, rsub = lane & 7, csub = lane >> 3;
  const bool last = 8 * (NT - 1) + rsub < nrow;
  const double* P = A + csub * lda + rsub;
  x += csub;
#pragma unroll
  for (int k = 0; k < NT; ++k) y[k] = 0.0;
  int c = 0;
  for (; c + 32 <= cols; c += 32, P += 32 * lda, x += 32) gemv_group<NT, true, kL2>(P, lda, 32, last, x, y);
  if (c < cols) gemv_group<NT, false, kL2>(P, lda, cols - c, last, x, y);
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    y[k] += __shfl_xor_sync(0xffffffffu, y[k], 8);
    y[k] += __shfl_xor_sync(0xffffffffu, y[k], 16);
  }
}
#define AFMM_TILES(nrow, CALL)   \
  switch (((nrow) + 7) >> 3) {   \
    case 1: CALL(1); break;      \
    case 2: CALL(2); break;      \
    case 3: CALL(3); break;      \
    case 4: CALL(4); break;      \
    default: CALL(5); break;     \
  }

constexpr int kUpWarps = 4, kDownWarps = 4;  // warps per box of the one-column sweeps

// M2M (src/AFMM2DTree.cpp:1129-1154): the box's outgoing charges L2P_b^T src_b
// over the row-major L2P copy; src_b = leaf charges, or the concatenated
// outgoing charges of children 0..3.  By one CTA: the warps share the node
// columns evenly, their sums are added in warp order.  ready() (by every
// thread, false: give up) comes between what is constant and the charges.
template <bool kL2, class Ready>
__device__ __forceinline__ void m2m_box(const LevelView& v, const double* __restrict__ src_all, int leaf, long b,
                                        Ready&& ready) {
  __shared__ double part[kUpWarps][40];
  const int r = v.rank[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = v.node_off[b + 1] - v.node_off[b];
  const double* src = src_all + (leaf ? v.leaf_start[b] : v.node_off[b]);
  const double* P = v.l2p_rm + v.l2p_off[b];  // (row c, column i) at i*r + c
  if (warp == 0) prefetch_l2_region(P, P + (long)n * r, lane);
  if (!ready() || r == 0) return;
  double* out = v.qhat + v.skel_off[b];
  const int c0 = warp * n / kUpWarps, c1 = (warp + 1) * n / kUpWarps;
  const int nch = (r + 39) / 40, step = ((r + nch - 1) / nch + 7) / 8 * 8;
  for (int i0 = 0; i0 < r; i0 += step) {
    const int nrow = min(step, r - i0);
#define AFMM_M2M(NT)                                                                              \
  {                                                                                               \
    double y[NT];                                                                                 \
    gemv_panel<NT, kL2>(P + (long)c0 * r + i0, r, nrow, c1 - c0, src + c0, y);                    \
    _Pragma("unroll") for (int k = 0; k < NT; ++k) if (lane < 8) part[warp][8 * k + lane] = y[k]; \
  }
    AFMM_TILES(nrow, AFMM_M2M)
#undef AFMM_M2M
    __syncthreads();
    if ((int)threadIdx.x < nrow) {
      double s = part[0][threadIdx.x];
#pragma unroll
      for (int w = 1; w < kUpWarps; ++w) s += part[w][threadIdx.x];
      out[i0 + threadIdx.x] = s;
    }
    __syncthreads();
  }
}

// L2L (src/AFMM2DTree.cpp:1180-1197): t = L2P_b yhat_b over the column-major
// L2P, added to the children's incoming potentials (the box's nodes are rows of
// level j + 1), or written as the leaf's potentials.  By one CTA whose warps
// take the box's row panels in turn; ready() as in m2m_box.
template <bool kL2, class Ready>
__device__ __forceinline__ void l2l_box(const LevelView& v, double* __restrict__ child_yhat, double* __restrict__ ys,
                                        int leaf, long b, Ready&& ready) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = v.rank[b];
  const int n = v.node_off[b + 1] - v.node_off[b];
  const double* P = v.l2p + v.l2p_off[b];  // (row i, column c) at c*n + i
  const double* yb = v.yhat + v.skel_off[b];
  double* out = leaf ? ys + v.leaf_start[b] : child_yhat + v.node_off[b];
  const int per = kDownWarps * ((n + 40 * kDownWarps - 1) / (40 * kDownWarps));  // panels
  const int step = per > 0 ? ((n + per - 1) / per + 7) / 8 * 8 : 8;
  if (warp == 0) prefetch_l2_region(P, P + (long)n * r, lane);
  if (!ready()) return;
  for (int i0 = warp * step; i0 < n; i0 += kDownWarps * step) {
    const int nrow = min(step, n - i0);
#define AFMM_L2L(NT)                                                                                  \
  {                                                                                                   \
    double y[NT], c[NT];                                                                              \
    _Pragma("unroll") for (int k = 0; k < NT; ++k) /* (asked for beside the operator) */              \
      c[k] = !leaf && lane < 8 && 8 * k + lane < nrow ? ld_src<kL2>(out + i0 + 8 * k + lane) : 0.0;   \
    gemv_panel<NT, kL2>(P + i0, n, nrow, r, yb, y);                                                   \
    _Pragma("unroll") for (int k = 0; k < NT; ++k)                                                    \
      if (lane < 8 && 8 * k + lane < nrow) out[i0 + 8 * k + lane] = leaf ? y[k] : c[k] + y[k];        \
  }
    AFMM_TILES(nrow, AFMM_L2L)
#undef AFMM_L2L
  }
}

// M2L (src/AFMM2DTree.cpp:1156-1178) of one column from the stored blocks,
// every unordered pair of boxes once: the block of (c, b) is the transpose of
// that of (b, c), so box b reads its blocks with the boxes in its forward
// slots (inner 0..7, outer 0..11: the opposites of inner 8..15, outer 12..23)
// and gives the potentials of both sides: its own rows' to yhat, and those of
// its forward boxes, one value per column, to v.back, from where m2l_back_row
// adds them to their rows.  Half the bytes of reading every block.
constexpr int kForwardSlots = 20;
__host__ __device__ __forceinline__ int forward_slot(int f) { return f < 8 ? f : 8 + f; }    // f -> slot of the list
__host__ __device__ __forceinline__ int backward_slot(int f) { return f < 8 ? 8 + f : 20 + f; }  // its opposite

// What the M2L needs of a box in one piece of memory (made at setup): its
// forward columns -- those before slot f, first skeleton row of slot f's box
// -- and where the columns' sums go.
struct ForwardBox {
  int64_t first;  // of the box's blocks (m2l_off)
  int64_t sums;   // of its columns in v.back
  int32_t r, row0;
  int32_t skip;   // stored columns between the inner and the outer forward blocks
  int32_t col[kForwardSlots + 1], row[kForwardSlots];
  // By one warp.
  __device__ __forceinline__ void make(const LevelView& v, long b, int lane) {
    const int c = lane < kForwardSlots ? v.il[b * 40 + forward_slot(lane)] : -1;
    const int d = lane < 8 ? v.il[b * 40 + 8 + lane] : -1;
    const int rc = c >= 0 ? v.rank[c] : 0;
    int pre = rc, sk = d >= 0 ? v.rank[d] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += t;
      sk += __shfl_xor_sync(0xffffffffu, sk, o);
    }
    if (lane < kForwardSlots) {
      col[lane] = pre - rc;
      row[lane] = c >= 0 ? v.skel_off[c] : 0;
    }
    if (lane == kForwardSlots) col[kForwardSlots] = pre;
    if (lane == 0) {
      first = v.m2l_off[b];
      sums = v.back_off[b];
      r = v.rank[b];
      row0 = v.skel_off[b];
      skip = sk;
    }
  }
  // Slot of column c (< col[kForwardSlots]): the last one that starts at or before c.
  __device__ __forceinline__ int slot_of(int c) const {
    int lo = 0, hi = kForwardSlots - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (col[mid] <= c) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  }
};

constexpr int kPairWarps = 4;    // warps per box
constexpr int kPairCols = 128;   // columns a warp stages the charges of at once
constexpr int kPairRows = 1024;  // rows of a box at once
inline size_t m2l_pair_smem(int rmax) {
  return kPairWarps * kPairCols * 2 * sizeof(double) +
         (size_t)std::min(rmax, kPairRows) * (1 + kPairWarps) * sizeof(double);
}

// One group of (up to) 32 columns of m2l_pair_panel: P is the entry of the
// lane's first row in its first column.  Only the last tile can hold rows past
// the panel's end, and only a tail group (not FULL) columns past the panel's:
// what stands at sq past those is another panel's charge, or no charge at all
// (past the staged columns come the sums that other lanes are writing), and a
// zero entry does not cancel it when it is not finite, so it is not read.
template <bool Q32, int NT, bool FULL>
__device__ __forceinline__ double m2l_pair_group(const void* __restrict__ P, long r, int left, const double* sq,
                                                 bool last, const double (&qb)[NT], double (&y)[NT]) {
  const int lane = threadIdx.x & 31, rsub = lane & 7, csub = lane >> 3;
  double t[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const bool vc = FULL || 4 * j + csub < left;
    const double qc = vc ? sq[4 * j] : 0.0;
    double m[NT];
#pragma unroll
    for (int k = 0; k < NT; ++k) {
      const bool ok = (FULL || vc) && (k + 1 < NT || last);
      if (Q32) {
        const uint32_t u = ok ? __ldg((const uint32_t*)P + 4 * j * r + 8 * k) : 0x80000000u;
        m[k] = __hiloint2double(0x43300000, (int)u) - 4503601774854144.0;  // u - 2^31, exact
      } else {
        m[k] = ok ? __ldg((const double*)P + 4 * j * r + 8 * k) : 0.0;
      }
    }
    t[j] = 0.0;
#pragma unroll
    for (int k = 0; k < NT; ++k) {
      y[k] += m[k] * qc;
      t[j] += m[k] * qb[k];
    }
  }
  // sum over the eight row lanes; lane rsub keeps column 4 rsub + csub
#pragma unroll
  for (int h = 4; h > 0; h >>= 1)
#pragma unroll
    for (int j = 0; j < h; ++j) {
      const bool up = rsub & h;
      const double send = up ? t[j] : t[j + h], keep = up ? t[j + h] : t[j];
      t[j] = keep + __shfl_xor_sync(0xffffffffu, send, h);
    }
  return t[0];
}

// A row panel (NT tiles of 8 rows) of `cols` columns stored one after the
// other from `first` on: lane (rsub, csub) holds rows 8 k + rsub of columns
// 32 g + 4 j + csub, so that a lane sums its rows of a column and its columns
// of a row in registers, and 14 shuffles per 32 columns finish the columns'
// sums.
template <bool Q32, int NT>
__device__ __forceinline__ void m2l_pair_panel(const LevelView& v, long first, int r, int i0, int nrow, int cols,
                                               const double* sq, double* st, const double* sqb, double* yp) {
  const int lane = threadIdx.x & 31, rsub = lane & 7, csub = lane >> 3;
  constexpr int E = Q32 ? 4 : 8;
  double y[NT], qb[NT];
  const bool last = 8 * (NT - 1) + rsub < nrow;
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    y[k] = 0.0;
    qb[k] = k + 1 < NT || last ? sqb[i0 + 8 * k + rsub] : 0.0;
  }
  const char* P = (Q32 ? (const char*)v.m2l_q : (const char*)v.m2l) + (first + (long)csub * r + i0 + rsub) * E;
  int cg = 0;
  for (; cg + 32 <= cols; cg += 32, P += 32l * r * E) {
    const double t = m2l_pair_group<Q32, NT, true>(P, r, 32, sq + cg + csub, last, qb, y);
    double* o = st + cg + 4 * rsub + csub;
    *o = i0 == 0 ? t : *o + t;
  }
  if (cg < cols) {
    const double t = m2l_pair_group<Q32, NT, false>(P, r, cols - cg, sq + cg + csub, last, qb, y);
    double* o = st + cg + 4 * rsub + csub;
    if (cg + 4 * rsub + csub < cols) *o = i0 == 0 ? t : *o + t;
  }
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    y[k] += __shfl_xor_sync(0xffffffffu, y[k], 8);
    y[k] += __shfl_xor_sync(0xffffffffu, y[k], 16);
    if ((k + 1 < NT || last) && csub == 0) yp[i0 + 8 * k + rsub] += y[k];
  }
}

// One CTA of kPairWarps warps per box, the forward columns shared evenly by
// the warps, the rows in panels of up to 40; the warps meet only to add their
// sums of the box's rows (in warp order).  Q32: the 32-bit fixed-point blocks;
// (u - 2^31) is exact, and the block's power of two goes to the charge of a
// column and to its sum (both exact).  At its start a warp asks for the first
// `ahead` bytes of its columns in L2.
template <bool Q32, class Ready>
__device__ __forceinline__ void m2l_pair_box(const LevelView& v, long b, uint32_t ahead, unsigned char* smem,
                                             Ready&& ready) {
  __shared__ ForwardBox s_fb[kPairWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ForwardBox& fb = s_fb[warp];
  for (int i = lane; i < (int)(sizeof(ForwardBox) / 8); i += 32) ((int64_t*)&fb)[i] = ((const int64_t*)(v.fwd + b))[i];
  __syncwarp();
  const int r = fb.r;
  if (r == 0) return;
  const int C = fb.col[kForwardSlots], ca = fb.col[8];
  const long gap = (long)fb.skip * r, first = fb.first;
  const int w0 = (int)((long)warp * C / kPairWarps), w1 = (int)((long)(warp + 1) * C / kPairWarps);
  if (ahead && lane == 0 && w1 > w0) {
    const uintptr_t m = Q32 ? (uintptr_t)v.m2l_q : (uintptr_t)v.m2l, E = Q32 ? 4 : 8;
    const uintptr_t a = (m + (uintptr_t)(first + (long)w0 * r + (w0 >= ca ? gap : 0)) * E) & ~(uintptr_t)15;
    const uintptr_t n = min((uintptr_t)ahead, ((uintptr_t)(w1 - w0) * r * E + 15) & ~(uintptr_t)15);
    if (w0 >= ca || w1 <= ca) prefetch_l2_bulk(a, (uint32_t)n);
  }
  ready();  // (the charges' producers are done)
  const int nr = min(r, kPairRows);
  double* sqb = (double*)smem;        // the box's own charges
  double* yp = sqb + nr + warp * nr;  // the warp's sums of the box's rows
  double* sq = sqb + (1 + kPairWarps) * nr + warp * 2 * kPairCols;  // charges of the staged columns
  double* st = sq + kPairCols;                                       // their sums
  for (int R0 = 0; R0 < r; R0 += kPairRows) {
    const int R1 = min(r, R0 + kPairRows);
    for (int i = lane; i < R1 - R0; i += 32) {
      yp[i] = 0.0;
      if (warp == 0) sqb[i] = v.qhat[fb.row0 + R0 + i];
    }
    for (int c0 = w0, c1; c0 < w1 || c0 == w0; c0 = c1) {
      c1 = min(w1, c0 + kPairCols);
      for (int c = lane; c < kPairCols; c += 32) {
        double q = 0.0;
        if (c0 + c < c1) {
          const int f = fb.slot_of(c0 + c);
          q = v.qhat[fb.row[f] + (c0 + c - fb.col[f])];
          if (Q32) q *= v.m2l_dec[b * 40 + forward_slot(f)].x;
        }
        sq[c] = q;
      }
      if (c0 == w0) __syncthreads();  // sqb
      else __syncwarp();
      if (c0 == c1) break;  // (a warp without columns)
      // the inner and the outer forward blocks: each one contiguous region of the box's storage
      const int cut = max(c0, min(c1, ca));
      const int nch = (R1 - R0 + 39) / 40, step = ((R1 - R0 + nch - 1) / nch + 7) / 8 * 8;
      for (int part = 0; part < 2; ++part) {
        const int a = part ? cut : c0, n = (part ? c1 : cut) - a;
        if (n <= 0) continue;
        const long e0 = first + (long)a * r + (part ? gap : 0) + R0;
        for (int i0 = 0; i0 < R1 - R0; i0 += step) {
          const int nrow = min(step, R1 - R0 - i0);
#define AFMM_PANEL(NT) m2l_pair_panel<Q32, NT>(v, e0, r, i0, nrow, n, sq + (a - c0), st + (a - c0), sqb, yp)
          switch ((nrow + 7) >> 3) {
            case 1: AFMM_PANEL(1); break;
            case 2: AFMM_PANEL(2); break;
            case 3: AFMM_PANEL(3); break;
            case 4: AFMM_PANEL(4); break;
            default: AFMM_PANEL(5); break;
          }
#undef AFMM_PANEL
        }
      }
      __syncwarp();
      for (int c = c0 + lane; c < c1; c += 32) {
        double t = Q32 ? st[c - c0] * v.m2l_dec[b * 40 + forward_slot(fb.slot_of(c))].x : st[c - c0];
        if (R0 > 0) t += v.back[fb.sums + c];
        v.back[fb.sums + c] = t;
      }
      __syncwarp();
    }
    __syncthreads();
    for (int i = threadIdx.x; i < R1 - R0; i += 32 * kPairWarps) {
      double s = sqb[nr + i];
#pragma unroll
      for (int w = 1; w < kPairWarps; ++w) s += sqb[(1 + w) * nr + i];
      v.yhat[fb.row0 + R0 + i] = s;
    }
    __syncthreads();
  }
}

// Adds to yhat[row] what the boxes that have row's box in a forward slot
// worked out for it.
__device__ __forceinline__ void m2l_back_row(const LevelView& v, long row) {
  const int b = v.skel_box[row];
  const int64_t* src = v.back_src + (long)b * kForwardSlots;
  const long i = row - v.skel_off[b];
  double s = v.yhat[row], t[kForwardSlots];
#pragma unroll
  for (int f = 0; f < kForwardSlots; ++f) {
    const int64_t o = src[f];
    t[f] = o >= 0 ? v.back[o + i] : 0.0;
  }
#pragma unroll
  for (int f = 0; f < kForwardSlots; ++f) s += t[f];
  v.yhat[row] = s;
}

// Source slots of leaf b's near field (neighbours 0..7, then the leaf itself),
// fetched by warp 0 in one round of loads instead of a walk by one thread
// (nine dependent neighbour -> leaf lookups): lane s < 9 reads slot s, the
// existing slots keep their order (compacted by a ballot), and a slot's
// offset is the sum of units(count) = ceil(count / UNIT) over the existing
// slots before it.  In lane s: the source leaf c (-1: no neighbour), its
// compacted index m (-1 if none), start, count, offset; in every lane the
// number of existing slots ns and the total of their units.  Warp 0, all 32
// lanes, only.
struct NearSlots {
  long c;
  int m, start, cnt, off, total, ns;
};

template <int UNIT>
__device__ __forceinline__ NearSlots near_slots(const NearView& nv, long b, int lane) {
  NearSlots r;
  r.c = -1;
  r.start = 0;
  r.cnt = 0;
  if (lane < 9) {
    r.c = lane < 8 ? (long)nv.nbr[b * 8 + lane] : b;
    if (r.c >= 0) {
      r.start = nv.leaf_start[r.c];
      r.cnt = nv.leaf_cnt[r.c];
    }
  }
  const bool ok = lane < 9 && r.c >= 0;
  const unsigned valid = __ballot_sync(0xffffffffu, ok);
  const int u = ok ? (r.cnt + UNIT - 1) / UNIT : 0;
  int pre = u;  // inclusive prefix over lanes 0..lane
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, pre, o);
    if (lane >= o) pre += t;
  }
  r.off = pre - u;
  r.total = __shfl_sync(0xffffffffu, pre, 8);
  r.ns = __popc(valid);
  r.m = ok ? __popc(valid & ((1u << lane) - 1u)) : -1;
  return r;
}

// Source segments of a CTA's targets: points src[m] .. of the arrays, from
// position off[m] of the flat list on.  Their sums go to part dst[m] - 1
// (dst = 0: the targets themselves, kNoPart: nowhere), or, without dst, to
// their place in the flat list.
constexpr int kNoPart = 1 << 20;
struct PairSegs {
  const int *src, *off, *dst;
  int n, total;
};
// What the source and target points are (the near field: leaf points and
// sorted charges; the on-the-fly M2L: skeletons and outgoing charges).
struct PairPoints {
  const double2* xy;
  const double* q;
  double* part;     // sums of the sources' side: the flat list's,
  long stride = 0;  // or parts of `stride` values
};

// One block of J x 32 sources: lane l owns the sources f0 + l, f0 + 32 + l, ...
// of the flat list, and meets target (l + t) mod n at step t, so that in every
// step the lanes (of a group) hold different targets.  KIND: the block's
// sources are all targets too (0: their sums go to `self`), all of another set
// (1), or neither (2: some lanes take no part in the targets' sums).
template <class K, int J, int KIND>
__device__ __forceinline__ void pair_block(const PairPoints& P, const KernelParams& kp, const PairSegs& sg, int f0,
                                           int n, const double2* px, const double* pq, double* acc, double* self,
                                           bool add) {
  const int lane = threadIdx.x & 31;
  double2 x[J];
  double w[J], sum[J];
  int idx[J], dst[J];  // dst -1: unused lane
#pragma unroll
  for (int u = 0; u < J; ++u) {
    const int f = f0 + 32 * u + lane;
    const int g = min(f, sg.total - 1);  // lanes past the end repeat the last source, unused
    int m = 0;
    while (m + 1 < sg.n && g >= sg.off[m + 1]) ++m;
    idx[u] = sg.src[m] + (g - sg.off[m]);
    dst[u] = f < sg.total ? (sg.dst ? sg.dst[m] : 1) : -1;
    x[u] = P.xy[idx[u]];
    w[u] = P.q[idx[u]];
    sum[u] = 0.0;
    // (a lane without a part in the targets' sums adds 0 * 0 there: its charge may be infinite)
    if (KIND == 2 && dst[u] <= 0) w[u] = 0.0;
  }
#pragma unroll 4
  for (int t = 0; t < n; ++t) {
    const double2 p = px[t];
    const double qi = pq[t];
    double a = KIND > 0 ? acc[t] : 0.0;
#pragma unroll
    for (int u = 0; u < J; ++u) {
      const double dx = x[u].x - p.x, dy = x[u].y - p.y;
      const double k = K::eval(dx * dx + dy * dy, kp);
      sum[u] += k * qi;
      if (KIND == 1) a += k * w[u];
      if (KIND == 2) a += (dst[u] > 0 ? k : 0.0) * w[u];
    }
    if (KIND > 0) {
      acc[t] = a;
      __syncwarp();  // the next lane takes the target over
    }
  }
#pragma unroll
  for (int u = 0; u < J; ++u) {
    if (dst[u] > 0 && dst[u] != kNoPart) {
      double* o = P.part + (sg.dst ? (long)(dst[u] - 1) * P.stride + idx[u] : f0 + 32 * u + lane);
      *o = add ? *o + sum[u] : sum[u];
    } else if (dst[u] == 0) self[f0 + 32 * u + lane] = sum[u];  // the targets come first in the flat list
  }
}

// Shared memory of pair_targets, for n targets.
struct PairSmem {
  double2* px;
  double *pq, *self, *accs;
  int row;
  __device__ __forceinline__ PairSmem(unsigned char* smem, int n) : row(near_row(n)) {
    px = (double2*)smem;
    pq = (double*)(px + row);
    self = pq + row;
    accs = self + n;
  }
};

// The sums of n targets (from point t0 on) against the sources of sg, and the
// sources' sums against the targets, by `warps` warps of the CTA that share
// the blocks of 32 sources evenly.  The caller's segments must be visible to
// every thread; nself: the leading sources that are the targets themselves
// (n or 0); add: the sources' sums are added to what their places hold.
// Afterwards pair_target_sum gives a target's sum.
template <class K>
__device__ __forceinline__ void pair_targets(const PairPoints& P, const KernelParams& kp, const PairSegs& sg, long t0,
                                             int n, int nself, int warps, const PairSmem& sm, bool add = false) {
  for (int t = threadIdx.x; t < sm.row; t += blockDim.x) {
    const int i = t % n;
    sm.px[t] = P.xy[t0 + i];
    sm.pq[t] = P.q[t0 + i];
  }
  for (int i = threadIdx.x; i < warps * sm.row; i += blockDim.x) sm.accs[i] = 0.0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < warps) {
    const int l0 = n >= 32 ? lane : lane % n;  // the lane's first target
    double* acc = sm.accs + warp * sm.row + (n >= 32 ? 0 : 2 * (lane - l0)) + l0;
    const int nblk = (sg.total + 31) >> 5, b1 = (warp + 1) * nblk / warps;
#define AFMM_PAIR(J, KIND) pair_block<K, J, KIND>(P, kp, sg, 32 * k, n, sm.px + l0, sm.pq + l0, acc, sm.self, add)
    for (int k = warp * nblk / warps; k < b1;) {
      const int nb = min(kNearJ, b1 - k);
      const int kind = 32 * (k + nb) <= nself ? 0 : (32 * k >= nself && 32 * (k + nb) <= sg.total ? 1 : 2);
      if (nb == 2) {
        if (kind == 0) AFMM_PAIR(2, 0);
        else if (kind == 1) AFMM_PAIR(2, 1);
        else AFMM_PAIR(2, 2);
      } else {
        if (kind == 0) AFMM_PAIR(1, 0);
        else if (kind == 1) AFMM_PAIR(1, 1);
        else AFMM_PAIR(1, 2);
      }
      k += nb;
    }
#undef AFMM_PAIR
  }
  __syncthreads();
}

// Target i's sum over the sources that are not targets: the warps' sums in
// warp order (each the sum of its lane groups' rows and of their two laps).
__device__ __forceinline__ double pair_target_sum(const PairSmem& sm, int n, int warps, int i, double v) {
  for (int x = 0; x < warps; ++x) {
    const double* r = sm.accs + x * sm.row + i;
    if (n >= 32) v += i < 32 ? r[0] + r[n] : r[0];
    else
      for (int c = 0; c < sm.row; c += 2 * n) v += r[c] + r[c + n];
  }
  return v;
}

// Source leaves of leaf b in the pairwise near fields: the leaf itself, then its
// neighbours in slots 0..3.  Per segment the first point, the position in the
// flat list, and what the sums go to (PairSegs); whether slots 4..7 exist.
struct NearSources {
  int src[5], off[6], dst[5], back[4], ns;
  // By one warp.
  __device__ __forceinline__ void make(const NearView& nv, long b, int lane) {
    // lane 0: the leaf; lanes 1..4: neighbour slots 0..3; lanes 5..8: slots 4..7
    long c = -1;
    int cnt = 0, start = 0;
    if (lane < 9) {
      c = lane == 0 ? b : (long)nv.nbr[b * 8 + lane - 1];
      if (c >= 0 && lane < 5) {
        start = nv.leaf_start[c];
        cnt = nv.leaf_cnt[c];
      }
    }
    const unsigned valid = __ballot_sync(0xffffffffu, lane < 5 && c >= 0);
    int pre = cnt;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += t;
    }
    if (lane < 5 && c >= 0) {
      const int m = __popc(valid & ((1u << lane) - 1u));
      src[m] = start;
      off[m] = pre - cnt;
      // (a leaf outside the shard gets no sums; part 0 is the leaf's own)
      dst[m] = lane == 0 ? 0 : (c >= nv.leaf0 && c < nv.leaf0 + nv.nleaf ? lane + 1 : kNoPart);
    }
    if (lane == 4) {
      ns = __popc(valid);
      off[__popc(valid)] = pre;
    }
    if (lane >= 5 && lane < 9) back[lane - 5] = c >= 0;
  }
};

// Near field (src/AFMM2DTree.cpp:1199-1213) of leaf b, kernel evaluated on the
// fly, every unordered pair of leaves once: K(x, y) depends on |x - y| only, so
// the pairs of leaf b with the neighbours in slots 0..3 give both leaves' sums
// (slots 4..7 are their opposites: those pairs belong to the neighbours), and
// with itself the leaf's own.  Per point nv.part[0] takes the leaf's own
// work and part[1 + s] what its neighbour in slot 4 + s worked out for it
// (zero without one); the scatter adds the five in that order.  An entry costs
// 12 to 25 FP64 operations and about as many integer ones, its use two, so
// working it out once for both leaves (5/9 of the entries) pays for the target
// sums that go from lane to lane through shared memory (four cycles of 18 an
// entry pair takes there).  What bounds it now is issue (62% of the slots,
// FP64 pipe 53% busy) and the polynomials' dependent steps: 80 registers (24
// warps an SM) measured faster than 102 or 64.  Near field at 1,048,576 uniform
// points, one CTA per leaf, all nine source leaves before -> now: log 1.34 ->
// 0.83 ms, Gaussian 1.03 -> 0.67, 1/r (mixture) 0.64 -> 0.42; 100,003 points of
// scaled 1/r (M = 100) 0.63 -> 0.40.  Run by one CTA of near_warps(nmax) warps
// that share the blocks of 32 source points evenly (more may be present); the
// sums of the warps are added in warp order.
template <class K>
__device__ __forceinline__ void near_leaf(const NearView& nv, const KernelParams& kp, const double* __restrict__ qs,
                                          int warps, long b, unsigned char* smem) {
  __shared__ NearSources src;
  const int n = nv.leaf_cnt[b];
  const int s0 = nv.leaf_start[b];
  const bool own = b >= nv.leaf0 && b < nv.leaf0 + nv.nleaf;
  if (threadIdx.x < 32) src.make(nv, b, threadIdx.x);
  const PairSmem sm(smem, n);
  __syncthreads();
  pair_targets<K>(PairPoints{nv.pts, qs, nv.part, nv.n}, kp,
                  PairSegs{src.src, src.off, src.dst, src.ns, src.off[src.ns]}, s0, n, n, warps, sm);
  if (!own) return;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    nv.part[s0 + i] = pair_target_sum(sm, n, warps, i, sm.self[i]);
    for (int s = 0; s < 4; ++s)
      if (!src.back[s]) nv.part[(size_t)(1 + s) * nv.n + s0 + i] = 0.0;
  }
}

// Sum of the near field's parts of sorted point i.
__device__ __forceinline__ double near_sum(const double* __restrict__ part, long n, long i) {
  return (((part[i] + part[n + i]) + part[2 * n + i]) + part[3 * n + i]) + part[4 * n + i];
}

void build_lists(int j, long nbox, int32_t* nbr, int32_t* il, cudaStream_t s);
// map[off[b] + l] = b for l < off[b+1] - off[b]
void fill_box_map(const int32_t* off, long nbox, int32_t* map, cudaStream_t s);
// iperm[perm[i]] = i
void invert_permutation(const int64_t* perm, int n, int32_t* iperm, cudaStream_t s);
// out[t] = pts[ids[t]]
void gather_points(const double2* pts, const int32_t* ids, long n, double2* out, cudaStream_t s);
void m2l_assemble(const LevelView& v, const KernelParams& kp, cudaStream_t s);
// 32-bit fixed-point copy of the stored FP64 blocks (m2l_q, m2l_dec).
void m2l_compress(const LevelView& v, cudaStream_t s);
// Forward columns of a level's boxes (v.fwd, v.back_src).
void forward_boxes(const LevelView& v, cudaStream_t s);
void l2p_transpose(const LevelView& v, const double* cm, double* rm, cudaStream_t s);
void matvec_fp64(const MatvecPlan& p, const double* q, double* y, cudaStream_t s, StageTimer* tm, int64_t* launches);
// One-column M2L of every level in FP64: the stored blocks, or m2l_apply_otf
// when no blocks are stored.  These return the launches made.
int m2l_apply(const MatvecPlan& p, cudaStream_t s);
// M2L of the given levels from the stored blocks, 32-bit fixed point (q32)
// or FP64, FP64 arithmetic.
int m2l_apply_stored(const MatvecPlan& p, const LevelSet& levels, bool q32, cudaStream_t s);
// M2L of the given levels with the entries evaluated on the fly in FP64 (mixed.cu).
int m2l_apply_otf(const MatvecPlan& p, const LevelSet& levels, cudaStream_t s);
// Their second launch: the sums that other boxes worked out (m2l_back_row).
int m2l_back(const LevelSet& ls, bool early, cudaStream_t s);
// The FP64 sweeps shared by both precisions (leaf charges qs in FP64).
void sweep_m2m(const MatvecPlan& p, const double* qs, cudaStream_t s, int64_t* launches);
void sweep_l2l(const MatvecPlan& p, double* ys, cudaStream_t s, int64_t* launches);

}  // namespace afmm
