// K2 (interaction lists), K5 (M2L blocks) and the FP64 matvec sweeps
// K6-K10 (gather, M2M, M2L, L2L, near field, scatter).
#include <algorithm>

#include "afmm_internal.cuh"
#include "fmm.cuh"
#include "kernel_table.cuh"

namespace afmm {

// ----------------------------------------------------------------- lists
// Closed form of the reference's parent-to-child recurrence
// (src/AFMM2DTree.cpp:65-967).  Box k at level j sits at grid cell (ix, iy)
// whose bits are the base-4 digits of k read as child offsets
// 0:(0,0) 1:(1,0) 2:(1,1) 3:(0,1) (src/AFMM2DTree.cpp:978-986).  Slot s of
// ring m (m = 1 neighbours N0..N7, 2 inner I0..I15, 3 outer O0..O23) is the
// cell at the s-th offset counter-clockwise around the ring starting at
// (-m,-m).  It is set when the cell is inside the domain and, for ring 3,
// when its parent neighbours the box's parent (the recurrence only visits the
// children of the parent's neighbours).
__device__ __forceinline__ void ring_offset(int m, int s, int& dx, int& dy) {
  const int side = 2 * m, seg = s / side, t = s % side;
  if (seg == 0) { dx = -m + t; dy = -m; }
  else if (seg == 1) { dx = m; dy = -m + t; }
  else if (seg == 2) { dx = m - t; dy = m; }
  else { dx = -m; dy = m - t; }
}

// One thread per (box, slot of the 48 ring slots).
__global__ void k_lists(int j, long nbox, int32_t* nbr, int32_t* il) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nbox * 48) return;
  long k = t / 48;
  int s = (int)(t % 48);
  int m = s < 8 ? 1 : (s < 24 ? 2 : 3);
  int ss = s < 8 ? s : (s < 24 ? s - 8 : s - 24);
  int ix, iy, dx, dy;
  cell_of(k, j, ix, iy);
  ring_offset(m, ss, dx, dy);
  const int side = 1 << j;
  int cx = ix + dx, cy = iy + dy;
  bool ok = cx >= 0 && cy >= 0 && cx < side && cy < side;
  if (ok && m == 3) ok = abs((cx >> 1) - (ix >> 1)) <= 1 && abs((cy >> 1) - (iy >> 1)) <= 1;
  int32_t v = ok ? (int32_t)box_of(cx, cy, j) : -1;
  if (m == 1) nbr[k * 8 + ss] = v;
  else il[k * 40 + (s - 8)] = v;  // inner 0..15 then outer 0..23
}

void build_lists(int j, long nbox, int32_t* nbr, int32_t* il, cudaStream_t s) {
  long n = nbox * 48;
  k_lists<<<(int)((n + 255) / 256), 256, 0, s>>>(j, nbox, nbr, il);
  AFMM_LAUNCH_CHECK();
}

__global__ void k_fill_box_map(const int32_t* __restrict__ off, long nbox, int32_t* map) {
  long b = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbox) return;
  for (int32_t t = off[b]; t < off[b + 1]; ++t) map[t] = (int32_t)b;
}

__global__ void k_invert_perm(const int64_t* __restrict__ perm, int n, int32_t* iperm) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) iperm[perm[i]] = i;
}

__global__ void k_gather_points(const double2* __restrict__ pts, const int32_t* __restrict__ ids, long n,
                                double2* out) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) out[t] = pts[ids[t]];
}

void gather_points(const double2* pts, const int32_t* ids, long n, double2* out, cudaStream_t s) {
  if (n == 0) return;
  k_gather_points<<<(int)((n + 255) / 256), 256, 0, s>>>(pts, ids, n, out);
  AFMM_LAUNCH_CHECK();
}

void invert_permutation(const int64_t* perm, int n, int32_t* iperm, cudaStream_t s) {
  k_invert_perm<<<(n + 255) / 256, 256, 0, s>>>(perm, n, iperm);
  AFMM_LAUNCH_CHECK();
}

void fill_box_map(const int32_t* off, long nbox, int32_t* map, cudaStream_t s) {
  k_fill_box_map<<<(int)((nbox + 255) / 256), 256, 0, s>>>(off, nbox, map);
  AFMM_LAUNCH_CHECK();
}

// ------------------------------------------------------------ M2L blocks
// (k_m2l_assemble, fmm_k.cuh)
void m2l_assemble(const LevelView& v, const KernelParams& kp, cudaStream_t s) {
  kernel_table(kp.id).m2l_assemble(v, kp, s);
}

// 32-bit fixed-point copy of the FP64 blocks: per block a power-of-two scale
// 2^k with max|M| * 2^-k in [2^30, 2^31), entries rounded to the nearest
// multiple of 2^k (absolute error <= 2^-31 max|M|) and stored offset by 2^31
// as unsigned.  A block whose largest entry is 0 or below 2^-960 decodes to
// zeros; a block holding a non-finite entry decodes to NaN (as the FP64
// blocks would propagate it).  One CTA per box.
__global__ void __launch_bounds__(256) k_m2l_compress(LevelView v) {
  const long b = blockIdx.x;
  const int r = v.rank[b];
  __shared__ double red[8];
  __shared__ double2 s_dec;
  const double* M = v.m2l + v.m2l_off[b];
  uint32_t* Q = v.m2l_q + v.m2l_off[b];
  long off = 0;
  for (int s = 0; s < 40; ++s) {
    const int c = v.il[b * 40 + s];
    const int rc = (c >= 0 && r > 0) ? v.rank[c] : 0;
    const long n = (long)r * rc;
    if (n == 0) {
      if (threadIdx.x == 0) v.m2l_dec[b * 40 + s] = make_double2(0.0, 0.0);
      continue;
    }
    double mx = 0.0;
    bool bad = false;
    for (long e = threadIdx.x; e < n; e += blockDim.x) {
      const double x = M[off + e];
      bad |= !isfinite(x);
      mx = fmax(mx, fabs(x));
    }
    if (bad) mx = __longlong_as_double(0x7ff0000000000000ll);  // +inf
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, red[w]);
      int ex = 0;
      frexp(m, &ex);  // m in [2^(ex-1), 2^ex)
      const int k = ex - 31;
      if (!isfinite(m)) {
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        s_dec = make_double2(nan, nan);
      } else if (m == 0.0 || k < -960) {
        s_dec = make_double2(0.0, 0.0);
      } else {
        const double sc = scalbn(1.0, k);
        s_dec = make_double2(sc, -(4503601774854144.0 * sc));  // 2^52 + 2^31
      }
      v.m2l_dec[b * 40 + s] = s_dec;
    }
    __syncthreads();
    const double2 dec = s_dec;
    const bool zero = !(dec.x != 0.0) || !isfinite(dec.x);
    int ex = 0;
    if (!zero) frexp(dec.x, &ex);
    const int k = ex - 1;  // dec.x = 2^k
    for (long e = threadIdx.x; e < n; e += blockDim.x) {
      uint32_t u = 0x80000000u;
      if (!zero) {
        long long t = llrint(scalbn(M[off + e], -k)) + 0x80000000ll;
        t = t < 0 ? 0 : (t > 0xffffffffll ? 0xffffffffll : t);
        u = (uint32_t)t;
      }
      Q[off + e] = u;
    }
    off += n;
    __syncthreads();
  }
}

void m2l_compress(const LevelView& v, cudaStream_t s) {
  k_m2l_compress<<<(int)v.nbox, 256, 0, s>>>(v);
  AFMM_LAUNCH_CHECK();
}

// ---------------------------------------------------------------- sweeps
// qs[i] = q[perm[i]]  (src/AFMM2D.cpp:49-51)
__global__ void k_gather(const double* __restrict__ q, const int64_t* __restrict__ perm, int n, double* qs) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  dep_release();
  if (i < n) qs[i] = q[perm[i]];
}

// y[perm[i]] = ys[i] + near field  (src/AFMM2D.cpp:61-63); ys keeps the sum
// (afmm_eval_error reads it)
__global__ void k_scatter(double* __restrict__ ys, const double* __restrict__ part, const int64_t* __restrict__ perm,
                          int n, double* y) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v = ys[i] + near_sum(part, n, i);
  ys[i] = v;
  y[perm[i]] = v;
}

// Row-major copy of L2P (per box, r fastest) for the M2M sweep.
template <class T>
__global__ void k_l2p_transpose(LevelView v, const T* __restrict__ cm, T* rm) {
  const long b = blockIdx.x;
  const int r = v.rank[b];
  if (r == 0) return;
  const int n = v.node_off[b + 1] - v.node_off[b];
  const long o = v.l2p_off[b];
  for (int e = threadIdx.x; e < n * r; e += blockDim.x) {
    int i = e / r, c = e - i * r;
    rm[o + e] = cm[o + (long)c * n + i];
  }
}

void l2p_transpose(const LevelView& v, const double* cm, double* rm, cudaStream_t s) {
  k_l2p_transpose<double><<<(int)v.nbox, 256, 0, s>>>(v, cm, rm);
  AFMM_LAUNCH_CHECK();
}

// One-column M2L of every level in one launch, one CTA per box (m2l_pair_box,
// fmm.cuh: every unordered pair of boxes once), the upper levels' boxes with
// their larger ranks first.  1,048,576 uniform points, log, TOL 10 (2.3 GB of
// blocks): 0.95 ms with every block read by a warp per 32 rows -> 0.55, 4.2 TB/s
// of the 6.5 measured (fixed point 0.48); a third of a CTA's time is the latency
// of its tables and charges.  Two warps a box instead of four: 0.57, and 26
// instead of 19 us at 4,096 points; copies through shared memory (cp.async)
// instead of registers: 0.67.
template <bool Q32>
__global__ void __launch_bounds__(32 * kPairWarps, 6) k_m2l_pair(LevelSet ls) {
  extern __shared__ __align__(16) unsigned char smem[];
  const long g = blockIdx.x;
  int j = 0;
  while (j + 1 < ls.nlev && g >= ls.m0[j + 1]) ++j;
  const LevelView& v = ls.lv[j];
  const long t = g - ls.m0[j];
  dep_release();
  m2l_pair_box<Q32>(v, v.m2l_run ? (long)v.m2l_run[t] : t, ls.pf_ahead, smem, [] { dep_wait(); });
}

__global__ void __launch_bounds__(128) k_forward_boxes(LevelView v) {
  const long b = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (b < v.nbox) v.fwd[b].make(v, b, threadIdx.x & 31);
}

__global__ void __launch_bounds__(128) k_back_src(LevelView v) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= v.nbox * kForwardSlots) return;
  const int f = (int)(t % kForwardSlots);
  const int c = v.il[t / kForwardSlots * 40 + backward_slot(f)];
  v.back_src[t] = c >= 0 && v.rank[c] > 0 ? v.fwd[c].sums + v.fwd[c].col[f] : -1;
}

void forward_boxes(const LevelView& v, cudaStream_t s) {
  k_forward_boxes<<<(int)((v.nbox * 32 + 127) / 128), 128, 0, s>>>(v);
  AFMM_LAUNCH_CHECK();
  k_back_src<<<(int)((v.nbox * kForwardSlots + 127) / 128), 128, 0, s>>>(v);
  AFMM_LAUNCH_CHECK();
}

// The sums that other boxes worked out, added to every level's rows.
__global__ void __launch_bounds__(256) k_m2l_back(LevelSet ls) {
  dep_release();
  dep_wait();
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= ls.row0[ls.nlev]) return;
  int j = 0;
  while (j + 1 < ls.nlev && g >= ls.row0[j + 1]) ++j;
  m2l_back_row(ls.lv[j], g - ls.row0[j]);
}

// One-column M2M and L2L of a level, one CTA per box (m2m_box, l2l_box): a
// level is then two latencies deep (tables, then the box's whole operator and
// its vector at once) instead of a warp per 32 rows that walks the operator.
// M2M + L2L as dependent launches: 1,048,576 uniform points (log, TOL 10) 0.39 ->
// 0.26 ms, 300,000 (mixture, 1/r) 0.29 -> 0.16, 4,096 43 -> 21 us.
__global__ void __launch_bounds__(32 * kUpWarps, 20 / kUpWarps) k_m2m_box(LevelView v, const double* __restrict__ src_all,
                                                                 int leaf) {
  dep_release();
  m2m_box<false>(v, src_all, leaf, blockIdx.x, [] {
    dep_wait();
    return true;
  });
}

__global__ void __launch_bounds__(32 * kDownWarps, 28 / kDownWarps) k_l2l_box(LevelView v, double* __restrict__ child_yhat,
                                                                 double* __restrict__ ys, int leaf) {
  dep_release();
  l2l_box<false>(v, child_yhat, ys, leaf, v.box0 + blockIdx.x, [] {
    dep_wait();
    return true;
  });
}

void sweep_m2m(const MatvecPlan& p, const double* qs, cudaStream_t s, int64_t* launches) {
  for (int j = p.L; j >= 2; --j) {
    const LevelView& v = p.lv[j];
    if (v.nrows == 0) continue;
    launch_dependent(p.small(), k_m2m_box, v.nbox, 32 * kUpWarps, 0, s, v, j == p.L ? qs : p.lv[j + 1].qhat, j == p.L);
    ++*launches;
  }
}

void sweep_l2l(const MatvecPlan& p, double* ys, cudaStream_t s, int64_t* launches) {
  for (int j = 2; j <= p.L; ++j) {
    const LevelView& v = p.lv_down[j];  // a shard's subtrees at the sharded levels
    if (v.nnodes == 0) continue;
    launch_dependent(p.small(), k_l2l_box, v.nrun, 32 * kDownWarps, 0, s, v, j < p.L ? p.lv[j + 1].yhat : nullptr, ys, j == p.L);
    ++*launches;
  }
}

int m2l_back(const LevelSet& ls, bool early, cudaStream_t s) {
  const long rows = ls.row0[ls.nlev];
  launch_dependent(early, k_m2l_back, (rows + 255) / 256, 256, 0, s, ls);
  return 1;
}

int m2l_apply(const MatvecPlan& p, cudaStream_t s) {
  const long rows = p.levels.row0[p.levels.nlev];
  if (rows == 0) return 0;
  if (p.levels.lv[0].m2l == nullptr) return m2l_apply_otf(p, p.levels, s);  // blocks not stored: entries on the fly
  return m2l_apply_stored(p, p.levels_m2l, false, s);  // a shard's boxes at the sharded levels
}

int m2l_apply_stored(const MatvecPlan& p, const LevelSet& levels, bool q32, cudaStream_t s) {
  LevelSet ls = levels;
  ls.pf_ahead = p.tune.pf_fp64;
  const long boxes = ls.m0[ls.nlev];
  if (boxes == 0 || ls.row0[ls.nlev] == 0) return 0;
  if (q32 && ls.lv[0].m2l_q == nullptr) throw Error{AFMM_BAD_ARG, "no fixed-point M2L blocks stored"};
  if (!q32 && ls.lv[0].m2l == nullptr) throw Error{AFMM_BAD_ARG, "no M2L blocks stored"};
  const size_t smem = m2l_pair_smem(*std::max_element(p.rmax, p.rmax + kMaxLevels));
  auto fn = q32 ? k_m2l_pair<true> : k_m2l_pair<false>;
  allow_smem(fn, smem);
  launch_dependent(p.small(), fn, boxes, 32 * kPairWarps, smem, s, ls);
  return 1 + m2l_back(ls, p.small(), s);
}

void matvec_fp64(const MatvecPlan& p, const double* q, double* y, cudaStream_t s, StageTimer* tm, int64_t* launches) {
  const int N = p.N;
  const int gb = (N + 255) / 256;
  if (tm) tm->mark(s, "gather");
  if (p.shard_count > 1) {
    AFMM_CUDA(cudaMemsetAsync(p.ys, 0, sizeof(double) * (size_t)N, s));
    AFMM_CUDA(cudaMemsetAsync(p.near.part, 0, sizeof(double) * kNearParts * (size_t)N, s));
  }
  k_gather<<<gb, 256, 0, s>>>(q, p.perm, N, p.qs);
  AFMM_LAUNCH_CHECK();
  ++*launches;
  beside_near(
      p, s, tm,
      [&](cudaStream_t st) {
        kernel_table(p.kp.id).p2p64(p.near_own, p.kp, p.qs, st);
        ++*launches;
      },
      [&](cudaStream_t st) {
        if (tm) tm->mark(st, "m2m");
        sweep_m2m(p, p.qs, st, launches);
        if (tm) tm->mark(st, "m2l");
        *launches += m2l_apply(p, st);
        if (tm) tm->mark(st, "l2l");
        sweep_l2l(p, p.ys, st, launches);
      });
  if (tm) tm->mark(s, "scatter");
  k_scatter<<<gb, 256, 0, s>>>(p.ys, p.near.part, p.perm, N, y);
  AFMM_LAUNCH_CHECK();
  ++*launches;
  if (tm) tm->mark(s, "end");
}

}  // namespace afmm
