// Many independent problems in fused launches (one launch per stage across
// all problems, each sweep over the levels one persistent launch, captured in
// one CUDA graph).  Each output row is computed by
// the same device functions as the single-problem FP64 path (fmm.cuh), so
// every problem's result is bit-identical to its own FP64 matvec.
#include <algorithm>

#include "kernel_table.cuh"
#include "set.cuh"

namespace afmm {

namespace {

// qs_p[i] = q[off[p] + perm_p[i]]  (src/AFMM2D.cpp:49-51 per problem)
__global__ void k_set_gather(SetDev d, SetSegs sg, const double* __restrict__ q) {
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= sg.total) return;
  const int s = seg_of(sg, g);
  const int p = sg.prob[s];
  const long i = g - sg.first[s];
  d.qs[p][i] = q[d.off[p] + d.perm[p][i]];
}

// y[off[p] + perm_p[i]] = ys_p[i] + near field  (src/AFMM2D.cpp:61-63 per problem)
__global__ void k_set_scatter(SetDev d, SetSegs sg, double* __restrict__ y) {
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= sg.total) return;
  const int s = seg_of(sg, g);
  const int p = sg.prob[s];
  const long i = g - sg.first[s];
  const double v = d.ys[p][i] + near_sum(d.nv[p].part, d.nv[p].n, i);
  d.ys[p][i] = v;
  y[d.off[p] + d.perm[p][i]] = v;
}

// ------------------------------------------------ persistent sweeps
// The M2M of every level of every problem runs in one launch (the up-sweep),
// and so does the L2L (the down-sweep).  Items are boxes, listed by depth in
// dependency order (M2M: each problem's leaf level first; L2L: level 2 first);
// a CTA takes the next box from a ticket counter, waits until the level that it
// reads has been published (per problem and level
// counters of boxes), computes it as the FP64 path does (same bits) and
// publishes it.  An item only waits for items earlier in
// the list, which CTAs already running hold, so the sweep cannot deadlock;
// each wait is still bounded in time, and a wait that gives up sets
// sync.err, makes every other wait give up and ends the launch early.

constexpr unsigned long long kWaitNs = 2000000000ull;  // 2 s of device time per wait

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// One thread waits until *c >= need; false if it gave up (time limit, or
// another wait gave up first).
__device__ bool wait_published(const int* c, long need, int* err) {
  if (ld_acquire(c) >= need) return true;
  const unsigned long long t0 = global_ns();
  for (int it = 0; it < (1 << 26); ++it) {
    __nanosleep(128);
    if (ld_acquire(c) >= need) return true;
    if (*(volatile int*)err) return false;
    if (global_ns() - t0 > kWaitNs) break;
  }
  atomicExch(err, 1);
  return false;
}

// Publishes the box that the CTA has just written.
__device__ __forceinline__ void publish_box(int* done) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(done, 1);
  }
}

// The next item of a sweep for the calling CTA (all threads), or -1.
__device__ __forceinline__ int next_item(int* ticket, int nitems, int* s_item) {
  __syncthreads();  // every thread has read the previous item
  if (threadIdx.x == 0) *s_item = atomicAdd(ticket, 1);
  __syncthreads();
  const int it = *s_item;
  return it < nitems ? it : -1;
}

// Up-sweep: M2M of every problem from its leaf level up to level 2.  A
// non-leaf level reads the outgoing charges of the level below.
__global__ void __launch_bounds__(32 * kUpWarps, 20 / kUpWarps) k_set_up(SetDev d, SweepPlan sw, SweepSync sy) {
  __shared__ int s_item, s_ok;
  for (int it; (it = next_item(sy.ticket, sw.nitems, &s_item)) >= 0;) {
    const SetSegs sg = sw.segs[sw.item_depth[it]];
    const long g = sw.item_first[it];
    const int s = seg_of(sg, g);
    const long pl = (long)sg.prob[s] * kMaxLevels + sg.level[s];
    const LevelView& v = d.lv[pl];
    const bool leaf = v.leaf_start != nullptr;
    m2m_box<true>(v, leaf ? d.qs[sg.prob[s]] : d.lv[pl + 1].qhat, leaf ? 1 : 0, g - sg.first[s], [&] {
      if (threadIdx.x == 0)
        s_ok = leaf || wait_published(sy.done_up + pl + 1, d.lv[pl + 1].nbox + sw.margin, sy.err);
      __syncthreads();
      return s_ok != 0;
    });
    if (!s_ok) return;  // the same in every thread of the CTA
    publish_box(sy.done_up + pl);
  }
}

// M2L of every level of every problem, one CTA per box, and the sums that
// other boxes worked out (skeleton rows).
__global__ void __launch_bounds__(32 * kPairWarps, 6) k_set_m2l(SetDev d, SetSegs sg) {
  extern __shared__ __align__(16) unsigned char smem[];
  const long g = blockIdx.x;
  const int s = seg_of(sg, g);
  const LevelView v = d.lv[(long)sg.prob[s] * kMaxLevels + sg.level[s]];
  m2l_pair_box<false>(v, g - sg.first[s], 12 * 1024, smem, [] {});
}

__global__ void __launch_bounds__(256) k_set_m2l_back(SetDev d, SetSegs sg) {
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= sg.total) return;
  const int s = seg_of(sg, g);
  m2l_back_row(d.lv[(long)sg.prob[s] * kMaxLevels + sg.level[s]], g - sg.first[s]);
}

// Down-sweep: L2L of every problem from level 2 down to its leaf level.
// Level j > 2 reads incoming potentials that the L2L of level j - 1 adds into.
__global__ void __launch_bounds__(32 * kDownWarps, 28 / kDownWarps) k_set_down(SetDev d, SweepPlan sw, SweepSync sy) {
  __shared__ int s_item, s_ok;
  for (int it; (it = next_item(sy.ticket + 1, sw.nitems, &s_item)) >= 0;) {
    const SetSegs sg = sw.segs[sw.item_depth[it]];
    const long g = sw.item_first[it];
    const int s = seg_of(sg, g);
    const long pl = (long)sg.prob[s] * kMaxLevels + sg.level[s];
    const LevelView& v = d.lv[pl];
    const bool leaf = v.leaf_start != nullptr;
    l2l_box<true>(v, leaf ? nullptr : d.lv[pl + 1].yhat, d.ys[sg.prob[s]], leaf ? 1 : 0, g - sg.first[s], [&] {
      if (threadIdx.x == 0)
        s_ok = sg.level[s] == 2 || wait_published(sy.done_dn + pl - 1, d.lv[pl - 1].nbox + sw.margin, sy.err);
      __syncthreads();
      return s_ok != 0;
    });
    if (!s_ok) return;  // the same in every thread of the CTA
    publish_box(sy.done_dn + pl);
  }
}

struct SegBuilder {
  std::vector<int64_t> first{0};
  std::vector<int32_t> prob, level;
  void add(int p, int j, long count) {
    if (count <= 0) return;
    prob.push_back(p);
    level.push_back(j);
    first.push_back(first.back() + count);
  }
  SetSegs upload(DevArena& arena, cudaStream_t s) const {
    SetSegs sg;
    sg.n = (int)prob.size();
    sg.total = first.back();
    int64_t* f = arena.alloc<int64_t>(first.size());
    int32_t* pr = arena.alloc<int32_t>(std::max<size_t>(prob.size(), 1));
    int32_t* lv = arena.alloc<int32_t>(std::max<size_t>(level.size(), 1));
    AFMM_CUDA(cudaMemcpyAsync(f, first.data(), sizeof(int64_t) * first.size(), cudaMemcpyHostToDevice, s));
    if (!prob.empty()) {
      AFMM_CUDA(cudaMemcpyAsync(pr, prob.data(), sizeof(int32_t) * prob.size(), cudaMemcpyHostToDevice, s));
      AFMM_CUDA(cudaMemcpyAsync(lv, level.data(), sizeof(int32_t) * level.size(), cudaMemcpyHostToDevice, s));
    }
    AFMM_CUDA(cudaStreamSynchronize(s));
    sg.first = f;
    sg.prob = pr;
    sg.level = lv;
    return sg;
  }
};

inline int nb(long n, int t) { return (int)((n + t - 1) / t); }

template <class T>
T* upload(const std::vector<T>& h, DevArena& arena, cudaStream_t s) {
  T* d = arena.alloc<T>(std::max<size_t>(h.size(), 1));
  if (!h.empty()) AFMM_CUDA(cudaMemcpyAsync(d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, s));
  return d;
}

void record(SetPlan& sp, cudaStream_t s) {
  int n = 0, m = 0;
  auto mark = [&](const char* name) {
    if ((size_t)m == sp.marks.size()) {
      cudaEvent_t e;
      AFMM_CUDA(cudaEventCreate(&e));
      sp.marks.push_back({name, e});
    }
    // an external record becomes an event-record node of the graph
    AFMM_CUDA(cudaEventRecordWithFlags(sp.marks[m].second, s, cudaEventRecordExternal));
    ++m;
  };
  // the sweeps' tickets and counters start at zero in every replay
  AFMM_CUDA(cudaMemsetAsync(sp.sync.ticket, 0, sp.sync.bytes, s));
  mark("gather");
  k_set_gather<<<nb(sp.gather.total, 256), 256, 0, s>>>(sp.dev, sp.gather, sp.q);
  AFMM_LAUNCH_CHECK();
  ++n;
  // the near field beside the far field (lower-priority branch)
  AFMM_CUDA(cudaEventRecord(sp.ev_q, s));
  AFMM_CUDA(cudaStreamWaitEvent(sp.s_near, sp.ev_q, 0));
  AFMM_CUDA(cudaEventRecordWithFlags(sp.near_mark[0], sp.s_near, cudaEventRecordExternal));
  kernel_table(sp.kernel_id).set_p2p_run(sp, sp.s_near);
  AFMM_CUDA(cudaEventRecordWithFlags(sp.near_mark[1], sp.s_near, cudaEventRecordExternal));
  AFMM_CUDA(cudaEventRecord(sp.ev_near, sp.s_near));
  ++n;
  mark("m2m");
  if (sp.up.nitems > 0) {
    k_set_up<<<sp.up.grid, 32 * kUpWarps, 0, s>>>(sp.dev, sp.up, sp.sync);
    AFMM_LAUNCH_CHECK();
    ++n;
  }
  mark("m2l");
  if (sp.m2l.total > 0) {
    k_set_m2l<<<(int)sp.m2l_box.total, 32 * kPairWarps, sp.m2l_smem, s>>>(sp.dev, sp.m2l_box);
    AFMM_LAUNCH_CHECK();
    k_set_m2l_back<<<nb(sp.m2l.total, 256), 256, 0, s>>>(sp.dev, sp.m2l);
    AFMM_LAUNCH_CHECK();
    n += 2;
  }
  mark("l2l");
  if (sp.down.nitems > 0) {
    k_set_down<<<sp.down.grid, 32 * kDownWarps, 0, s>>>(sp.dev, sp.down, sp.sync);
    AFMM_LAUNCH_CHECK();
    ++n;
  }
  mark("p2p");  // the wait for the near field's end
  AFMM_CUDA(cudaStreamWaitEvent(s, sp.ev_near, 0));
  mark("scatter");
  k_set_scatter<<<nb(sp.gather.total, 256), 256, 0, s>>>(sp.dev, sp.gather, sp.y);
  AFMM_LAUNCH_CHECK();
  ++n;
  mark("end");
  AFMM_CUDA(cudaMemcpyAsync(sp.h_err, sp.sync.err, sizeof(int), cudaMemcpyDeviceToHost, s));
  sp.launches_per_matvec = n;
}

}  // namespace

void set_build(SetPlan& sp, const std::vector<const MatvecPlan*>& probs, DevArena& arena, cudaStream_t s) {
  const int np = (int)probs.size();
  std::vector<LevelView> lv((size_t)np * kMaxLevels);
  std::vector<NearView> nv(np);
  std::vector<KernelParams> kp(np);
  std::vector<int> warps(np);
  std::vector<const int64_t*> perm(np);
  std::vector<double*> qs(np), ys(np);
  std::vector<int64_t> off(np + 1, 0);
  SegBuilder g, m2l, m2l_box, p2p;
  int rmax = 0;
  int maxL = 0;
  sp.p2p_threads = 0;
  sp.p2p_smem = 0;
  for (int p = 0; p < np; ++p) {
    const MatvecPlan& mp = *probs[p];
    for (int j = 0; j <= mp.L; ++j) lv[(size_t)p * kMaxLevels + j] = mp.lv[j];
    nv[p] = mp.near;
    kp[p] = mp.kp;
    warps[p] = near_warps(mp.near.nmax);
    perm[p] = mp.perm;
    qs[p] = mp.qs;
    ys[p] = mp.ys;
    off[p + 1] = off[p] + mp.N;
    g.add(p, 0, mp.N);
    for (int j = 2; j <= mp.L; ++j) m2l.add(p, j, mp.lv[j].nrows);
    for (int j = 2; j <= mp.L; ++j)
      if (mp.lv[j].nrows > 0) m2l_box.add(p, j, mp.lv[j].nbox);
    rmax = std::max(rmax, *std::max_element(mp.rmax, mp.rmax + kMaxLevels));
    p2p.add(p, mp.L, mp.near.nleaf);
    maxL = std::max(maxL, mp.L);
    sp.p2p_threads = std::max(sp.p2p_threads, 32 * warps[p]);
    sp.p2p_smem = std::max(sp.p2p_smem, near_smem(mp.near.nmax, warps[p]));
  }
  // M2M by depth below the leaf level; L2L by level from the top; each
  // sweep's items are the depth tables' boxes in that order
  sp.m2m.clear();
  sp.l2l.clear();
  std::vector<int32_t> up_d, dn_d;
  std::vector<int64_t> up_r, dn_r;
  auto tiles = [](long total, int depth, std::vector<int32_t>& dd, std::vector<int64_t>& rr) {
    for (long r = 0; r < total; ++r) {
      dd.push_back(depth);
      rr.push_back(r);
    }
  };
  for (int depth = 0; depth + 2 <= maxL; ++depth) {
    SegBuilder b;
    for (int p = 0; p < np; ++p) {
      const MatvecPlan& mp = *probs[p];
      const int j = mp.L - depth;
      if (j >= 2) b.add(p, j, mp.lv[j].nbox);
    }
    if (b.first.back() > 0) {
      tiles(b.first.back(), (int)sp.m2m.size(), up_d, up_r);
      sp.m2m.push_back(b.upload(arena, s));
    }
  }
  for (int j = 2; j <= maxL; ++j) {
    SegBuilder b;
    for (int p = 0; p < np; ++p) {
      const MatvecPlan& mp = *probs[p];
      if (j <= mp.L) b.add(p, j, mp.lv[j].nbox);
    }
    if (b.first.back() > 0) {
      tiles(b.first.back(), (int)sp.l2l.size(), dn_d, dn_r);
      sp.l2l.push_back(b.upload(arena, s));
    }
  }
  const int nsm = sm_count();
  int per_sm_up = 0, per_sm_dn = 0;
  AFMM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_up, k_set_up, 32 * kUpWarps, 0));
  AFMM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_dn, k_set_down, 32 * kDownWarps, 0));
  sp.up.segs = upload(sp.m2m, arena, s);
  sp.up.item_depth = upload(up_d, arena, s);
  sp.up.item_first = upload(up_r, arena, s);
  sp.up.nitems = (int)up_d.size();
  sp.up.grid = (int)std::min<long>(sp.up.nitems, (long)std::max(per_sm_up, 1) * nsm);
  sp.down.segs = upload(sp.l2l, arena, s);
  sp.down.item_depth = upload(dn_d, arena, s);
  sp.down.item_first = upload(dn_r, arena, s);
  sp.down.nitems = (int)dn_d.size();
  sp.down.grid = (int)std::min<long>(sp.down.nitems, (long)std::max(per_sm_dn, 1) * nsm);
  const size_t ncnt = (size_t)np * kMaxLevels;
  sp.sync.bytes = sizeof(int) * (3 + 2 * ncnt);
  sp.sync.ticket = arena.alloc<int>(3 + 2 * ncnt);
  sp.sync.err = sp.sync.ticket + 2;
  sp.sync.done_up = sp.sync.ticket + 3;
  sp.sync.done_dn = sp.sync.done_up + ncnt;
  if (!sp.h_err) {
    AFMM_CUDA(cudaHostAlloc((void**)&sp.h_err, sizeof(int), cudaHostAllocDefault));
    *sp.h_err = 0;
  }
  sp.gather = g.upload(arena, s);
  sp.m2l = m2l.upload(arena, s);
  sp.m2l_box = m2l_box.upload(arena, s);
  sp.m2l_smem = m2l_pair_smem(rmax);
  allow_smem(k_set_m2l, sp.m2l_smem);
  sp.p2p = p2p.upload(arena, s);
  sp.dev.nprob = np;
  sp.dev.lv = upload(lv, arena, s);
  sp.dev.nv = upload(nv, arena, s);
  sp.dev.kp = upload(kp, arena, s);
  sp.dev.p2p_warps = upload(warps, arena, s);
  sp.dev.perm = upload(perm, arena, s);
  sp.dev.qs = upload(qs, arena, s);
  sp.dev.ys = upload(ys, arena, s);
  sp.dev.off = upload(off, arena, s);
  sp.total_points = off[np];
  sp.q = arena.alloc<double>(off[np]);
  sp.y = arena.alloc<double>(off[np]);
  AFMM_CUDA(cudaStreamSynchronize(s));
  int least = 0, greatest = 0;
  AFMM_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
  AFMM_CUDA(cudaStreamCreateWithPriority(&sp.s_near, cudaStreamNonBlocking, least));
  AFMM_CUDA(cudaEventCreateWithFlags(&sp.ev_q, cudaEventDisableTiming));
  AFMM_CUDA(cudaEventCreateWithFlags(&sp.ev_near, cudaEventDisableTiming));
  for (cudaEvent_t& e : sp.near_mark) AFMM_CUDA(cudaEventCreate(&e));
  // kernel attributes are set before capture; then the graph is recorded once
  kernel_table(sp.kernel_id).set_p2p_prepare(sp.p2p_smem);
  set_recapture(sp, s);
}

void set_recapture(SetPlan& sp, cudaStream_t s) {
  if (sp.exec) AFMM_CUDA(cudaGraphExecDestroy(sp.exec));
  if (sp.graph) AFMM_CUDA(cudaGraphDestroy(sp.graph));
  sp.exec = nullptr;
  sp.graph = nullptr;
  AFMM_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  try {
    record(sp, s);
  } catch (...) {
    cudaGraph_t tmp = nullptr;
    cudaStreamEndCapture(s, &tmp);
    if (tmp) cudaGraphDestroy(tmp);
    cudaGetLastError();
    throw;
  }
  AFMM_CUDA(cudaStreamEndCapture(s, &sp.graph));
  AFMM_CUDA(cudaGraphInstantiate(&sp.exec, sp.graph, 0));
}

void set_matvec(SetPlan& sp, cudaStream_t s) { AFMM_CUDA(cudaGraphLaunch(sp.exec, s)); }

void set_stage_times(const SetPlan& sp, std::vector<std::pair<std::string, double>>& out) {
  out.clear();
  for (size_t i = 0; i + 1 < sp.marks.size(); ++i) {
    float ms = 0;
    AFMM_CUDA(cudaEventElapsedTime(&ms, sp.marks[i].second, sp.marks[i + 1].second));
    out.push_back({sp.marks[i].first, ms});
  }
  float ms = 0;
  AFMM_CUDA(cudaEventElapsedTime(&ms, sp.near_mark[0], sp.near_mark[1]));
  out.push_back({"p2p_kernel", ms});
}

void set_release(SetPlan& sp) {
  if (sp.h_err) cudaFreeHost(sp.h_err);
  sp.h_err = nullptr;
  if (sp.exec) cudaGraphExecDestroy(sp.exec);
  if (sp.graph) cudaGraphDestroy(sp.graph);
  for (auto& m : sp.marks) cudaEventDestroy(m.second);
  for (cudaEvent_t* e : {&sp.ev_q, &sp.ev_near, &sp.near_mark[0], &sp.near_mark[1]}) {
    if (*e) cudaEventDestroy(*e);
    *e = nullptr;
  }
  if (sp.s_near) cudaStreamDestroy(sp.s_near);
  sp.s_near = nullptr;
  sp.marks.clear();
  sp.exec = nullptr;
  sp.graph = nullptr;
}

}  // namespace afmm
