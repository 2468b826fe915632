// Kernel-templated stages of the single-RHS mixed path: M2L on the fly in
// FP64 and the FP32 near field, instantiated once per kernel functor by the
// kernel tables (kernel_table.cuh).
#pragma once
#include "mixed.cuh"

namespace afmm {

namespace mixed_detail {

// Threshold below which a near-field pair is re-evaluated in FP64.
template <class K>
__device__ __forceinline__ float fallback_r2(float span_b, float span_c) {
  float e = (span_b + span_c) * 0.0078125f;  // 2^-7 of the combined extent
  float t = e * e;
  if (K::id == AFMM_KERNEL_LOG) t = fmaxf(t, 4e-10f);
  return t;
}

// M2L on the fly in FP64 for every level, one CTA per box (upper levels
// first): the box's skeleton points against those of its forward
// interaction-list boxes, every entry worked out once for both (pair_targets,
// as the FP64 near field; the sums as in m2l_pair_box).  Issue-bound like it:
// 262,144 spiral points, log, TOL 12: 0.80 -> 0.35 ms (one thread per skeleton
// row, every entry worked out for both sides).
constexpr int kOtfWarps = 4;
template <class K>
__global__ void __launch_bounds__(32 * kOtfWarps, 6) k_m2l_otf(LevelSet ls, KernelParams kp) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ ForwardBox fb;
  const long g = blockIdx.x;
  int j = 0;
  while (j + 1 < ls.nlev && g >= ls.b0[j + 1]) ++j;
  const LevelView& v = ls.lv[j];
  const long b = g - ls.b0[j];
  if (threadIdx.x < sizeof(ForwardBox) / 8) ((int64_t*)&fb)[threadIdx.x] = ((const int64_t*)(v.fwd + b))[threadIdx.x];
  __syncthreads();
  const int r = fb.r;
  if (r == 0) return;
  const PairSegs sg{fb.row, fb.col, nullptr, kForwardSlots, fb.col[kForwardSlots]};
  for (int R0 = 0; R0 < r; R0 += kPairRows) {  // (one round unless the rank is beyond kPairRows)
    const int n = min(kPairRows, r - R0);
    const PairSmem sm(smem, n);
    pair_targets<K>(PairPoints{v.skel_xy, v.qhat, v.back + fb.sums}, kp, sg, fb.row0 + R0, n, 0, kOtfWarps, sm, R0 > 0);
    for (int i = threadIdx.x; i < n; i += 32 * kOtfWarps)
      v.yhat[fb.row0 + R0 + i] = pair_target_sum(sm, n, kOtfWarps, i, 0.0);
    __syncthreads();
  }
}

template <class K>
struct M2lOtfRun {
  static void run(const LevelSet& ls, int rmax, const KernelParams& kp, cudaStream_t s) {
    const long boxes = ls.b0[ls.nlev];
    if (boxes == 0) return;
    const size_t smem = near_smem(std::min(rmax, kPairRows), kOtfWarps);
    allow_smem(k_m2l_otf<K>, smem);
    same_carveout(k_m2l_otf<K>);
    k_m2l_otf<K><<<(int)boxes, 32 * kOtfWarps, smem, s>>>(ls, kp);
    AFMM_LAUNCH_CHECK();
  }
};

// Kernel entry of a close pair in FP64 from the exact coordinates; a point
// with itself (the diagonal) takes the kernel's value at zero distance
// without any FP64 work, so the self-interaction costs no divergent branch.
template <class K>
__device__ __noinline__ float near_pair(const NearView& nv, const KernelParams& kp, int p, int q) {
  if (p == q) return (float)K::at_zero(kp);
  const double2 a = nv.pts[p], c = nv.pts[q];
  return (float)K::eval_exact(r2_exact(a.x, a.y, c.x, c.y), kp);
}

// Near field in FP32 from leaf-relative coordinates.  One CTA per leaf; all
// source leaves (neighbours 0..7, then the leaf) are staged in shared memory
// at once, with each source leaf's anchor offset folded in FP64; each thread
// owns one target and sums all of its source leaves (the FP32 entries are
// cheap, so splitting the leaves over thread groups only adds imbalance and a
// reduction: 1.12 vs 1.62 ms at 1M uniform points, log), FP32 partial sums
// per source leaf added in FP64.  Issue-bound: a source is one 16-byte load,
// and the rare close pairs' FP64 form is a call (1M points: log 1.11 -> 0.95 ms,
// Gaussian 0.93 -> 0.74; 100,003 scaled 1/r, M = 100, 0.75 -> 0.64, with its
// divisions by powers of two as scalings).  Writes the sums of leaf b's points to
// `out`; the scatter adds them to the far field's.
template <class K>
__global__ void k_p2p32(NearView nv, KernelParams kp, const float* __restrict__ qs32, double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_src[9], s_cnt[9], s_off[10], s_ns;
  __shared__ float s_dx[9], s_dy[9], s_thr[9];
  const long b = nv.leaf0 + blockIdx.x;
  const int n = nv.leaf_cnt[b];
  const int s0 = nv.leaf_start[b];
  const float a32 = (float)kp.a, p32 = (float)kp.param;
  if (threadIdx.x < 32) {
    const NearSlots sl = near_slots<1>(nv, b, threadIdx.x);
    if (sl.m >= 0) {
      const double2 ab = nv.anchor[b], ac = nv.anchor[sl.c];
      s_src[sl.m] = sl.start;
      s_cnt[sl.m] = sl.cnt;
      s_off[sl.m] = sl.off;
      s_dx[sl.m] = (float)(ab.x - ac.x);
      s_dy[sl.m] = (float)(ab.y - ac.y);
      s_thr[sl.m] = fallback_r2<K>(nv.span[b], nv.span[sl.c]);
    }
    if (threadIdx.x == 0) {
      s_off[sl.ns] = sl.total;
      s_ns = sl.ns;
    }
  }
  __syncthreads();
  const int ns = s_ns;
  float4* sx = (float4*)smem;  // x, y, charge
  for (int m = 0; m < ns; ++m)
    for (int t = threadIdx.x; t < s_cnt[m]; t += blockDim.x) {
      const float2 p = nv.rel[s_src[m] + t];
      sx[s_off[m] + t] = make_float4(p.x, p.y, qs32[s_src[m] + t], 0.0f);
    }
  __syncthreads();
  const int i = threadIdx.x;
  double acc = 0.0;
  if (i < n) {
    const float2 xi = nv.rel[s0 + i];
    for (int m = 0; m < ns; ++m) {
      const int o = s_off[m], nc = s_cnt[m];
      const float ox = xi.x + s_dx[m], oy = xi.y + s_dy[m], thr = s_thr[m];
      float a0 = 0.0f, a1 = 0.0f;
      int t = 0;
      for (; t + 1 < nc; t += 2) {
        const float4 p0 = sx[o + t], p1 = sx[o + t + 1];
        const float dx0 = ox - p0.x, dy0 = oy - p0.y, dx1 = ox - p1.x, dy1 = oy - p1.y;
        const float R0 = fmaf(dx0, dx0, dy0 * dy0), R1 = fmaf(dx1, dx1, dy1 * dy1);
        float k0, k1;
        if (R0 < thr) k0 = near_pair<K>(nv, kp, s0 + i, s_src[m] + t);
        else k0 = K::eval32(R0, a32, p32);
        if (R1 < thr) k1 = near_pair<K>(nv, kp, s0 + i, s_src[m] + t + 1);
        else k1 = K::eval32(R1, a32, p32);
        a0 = fmaf(k0, p0.z, a0);
        a1 = fmaf(k1, p1.z, a1);
      }
      if (t < nc) {
        const float4 p0 = sx[o + t];
        const float dx0 = ox - p0.x, dy0 = oy - p0.y;
        const float R0 = fmaf(dx0, dx0, dy0 * dy0);
        float k0;
        if (R0 < thr) k0 = near_pair<K>(nv, kp, s0 + i, s_src[m] + t);
        else k0 = K::eval32(R0, a32, p32);
        a0 = fmaf(k0, p0.z, a0);
      }
      acc += (double)a0 + (double)a1;
    }
  }
  if (i < n) out[s0 + i] = acc;
}

template <class K>
struct P2p32Run {
  static void run(const NearView& nv, const KernelParams& kp, const float* qs32, double* out, cudaStream_t s) {
    const int threads = (nv.nmax + 31) / 32 * 32;
    const size_t smem = (size_t)9 * nv.nmax * sizeof(float4);
    allow_smem(k_p2p32<K>, smem);
    same_carveout(k_p2p32<K>);
    k_p2p32<K><<<(int)nv.nleaf, threads, smem, s>>>(nv, kp, qs32, out);
    AFMM_LAUNCH_CHECK();
  }
};

}  // namespace mixed_detail

}  // namespace afmm
