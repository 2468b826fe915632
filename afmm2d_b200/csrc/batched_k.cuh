// Kernel-templated stages of the batched (multi-RHS) path: M2L on the fly
// and the near fields, instantiated once per kernel functor by the kernel
// tables (kernel_table.cuh).
#pragma once
#include <algorithm>

#include "batched_common.cuh"
#include "mixed.cuh"

namespace afmm {

namespace batched_detail {

template <class K>
__device__ __forceinline__ float fallback_r2_b(float span_b, float span_c) {
  float e = (span_b + span_c) * 0.0078125f;
  float t = e * e;
  if (K::id == AFMM_KERNEL_LOG) t = fmaxf(t, 4e-10f);
  return t;
}

// TF32 MMA m16n8k8: lane l = 4g + t holds A[g][t], A[g+8][t], A[g][t+4],
// A[g+8][t+4]; B[t][g], B[t+4][g]; D[g][2t], D[g][2t+1], D[g+8][2t], D[g+8][2t+1].
__device__ __forceinline__ void mma_tf32_16x8x8(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// M2L on the fly with FP64 tensor-core tiles: one warp per row group (up to 8
// skeleton rows of one box).  For every interaction-list box and every 4 of
// its skeleton points, each lane evaluates the one FP64 entry it holds in the
// A fragment (row l/4, source l%4: no entry is evaluated twice) and the warp
// multiplies the 8x4 tile with the 4 x RC block of outgoing charges.
template <class K, int RC>
__global__ void __launch_bounds__(128) k_m2l_mma(LevelSet ls, KernelParams kp, const double* const* __restrict__ qhat_lv,
                                                 double* const* __restrict__ yhat_lv) {
  const long gw = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= ls.grp0[ls.nlev]) return;  // whole warps only
  int j = 0;
  while (j + 1 < ls.nlev && gw >= ls.grp0[j + 1]) ++j;
  const LevelView& v = ls.lv[j];
  const double* qh = qhat_lv[ls.src[j]];
  const long g = gw - ls.grp0[j];
  const int b = v.grp_box[g];
  const int r0 = v.grp_row[g];
  const int nv = min(8, v.skel_off[b] + v.rank[b] - r0);
  const int trow = lane >> 2, tsrc = lane & 3;
  const bool vrow = trow < nv;
  const double2 xi = vrow ? v.skel_xy[r0 + trow] : make_double2(0.0, 0.0);
  double c[RC / 8][2];
#pragma unroll
  for (int t = 0; t < RC / 8; ++t) c[t][0] = c[t][1] = 0.0;
  for (int s = 0; s < 40; ++s) {
    const int cb = v.il[(long)b * 40 + s];
    if (cb < 0) continue;
    const int rc = v.rank[cb];
    const int sc = v.skel_off[cb];
    for (int cc0 = 0; cc0 < rc; cc0 += 4) {
      const int cs = cc0 + tsrc;
      const bool vs = cs < rc;
      double a = 0.0;
      if (vrow && vs) {
        const double2 p = v.skel_xy[sc + cs];
        const double dx = xi.x - p.x, dy = xi.y - p.y;
        a = K::eval(dx * dx + dy * dy, kp);
      }
#pragma unroll
      for (int t = 0; t < RC / 8; ++t) {
        const double bq = vs ? qh[(long)(sc + cs) * RC + t * 8 + trow] : 0.0;
        mma_f64_8x8x4(c[t][0], c[t][1], a, bq);
      }
    }
  }
  if (vrow) {
    double* out = yhat_lv[ls.src[j]] + (long)(r0 + trow) * RC;
#pragma unroll
    for (int t = 0; t < RC / 8; ++t) {
      out[t * 8 + 2 * tsrc] = c[t][0];
      out[t * 8 + 2 * tsrc + 1] = c[t][1];
    }
  }
}

// TF32 high / low parts of an FP32 value by masking (the tensor cores read
// the top 19 bits of a TF32 operand): hi keeps 11 significant bits, lo the
// next 11 of the exact remainder; |x - hi - lo| <= 2^-21 |x|.
__device__ __forceinline__ void split_tf32_mask(float x, uint32_t& hi, uint32_t& lo) {
  hi = __float_as_uint(x) & 0xffffe000u;
  lo = __float_as_uint(x - __uint_as_float(hi)) & 0xffffe000u;
}

// Far-away stand-ins for padded source slots and absent targets: their
// entries are finite for every kernel and never below a fallback threshold;
// padded sources get zero charges and absent targets are not stored.
constexpr float kPadSrc = 1.0e15f, kPadTgt = -1.0e15f;

// Near field with TF32 tensor-core tiles in a three-term split
// (A_hi B_hi + A_hi B_lo + A_lo B_hi, ~FP32 accuracy).  One CTA per leaf, one
// warp per 32 targets (two 16 x 8 tiles sharing every charge fragment).  The
// source leaves (neighbours 0..7, then the leaf itself) are staged in shared
// memory in the target leaf's frame (each source leaf's anchor offset folded
// in FP64), padded to multiples of 8; the charges' interleaved TF32 high / low
// parts (split once per pass by the gather) come from L2, one 8-byte load per
// fragment element.  Each lane evaluates 8 FP32 entries per 8-source step; a
// warp vote sends the rare close pairs to the FP64 fallback.  The high*high
// products and the two correction products accumulate in separate FP32 tiles
// (independent MMA chains), which are added per source leaf into FP64 sums
// kept in shared memory.  Issue-bound; how the compiler orders the loads of a
// step among its entries depends on the registers it is told to keep to: 16
// columns for five CTAs an SM (1,048,576 points, log / Gaussian / 1/r 1.21 / 0.69 /
// 0.65 ms; four 1.31 / .75 / .73, six 1.59 / .85 / .70, left to it 1.32 / .77 / .73), 8
// columns left to it (.99 / .53 / .44; five .99 / .53 / .50).
template <class K, int RC>
__global__ void __launch_bounds__(128, RC == 16 ? 5 : 0) k_p2p_mma(NearView nv, KernelParams kp,
                                                                      const uint2* __restrict__ qhl,
                                                                      double* __restrict__ ys) {
  constexpr int NE = 2 * (RC / 8) * 4;  // FP64 sums per lane
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_src[9], s_cnt[9], s_coff[10], s_ns;
  __shared__ float s_dx[9], s_dy[9], s_thr[9];
  const long b = nv.leaf0 + blockIdx.x;
  const int n = nv.leaf_cnt[b];
  const int s0 = nv.leaf_start[b];
  const float a32 = (float)kp.a, p32 = (float)kp.param;
  if (threadIdx.x < 32) {
    const NearSlots sl = near_slots<8>(nv, b, threadIdx.x);
    if (sl.m >= 0) {
      const double2 ab = nv.anchor[b], ac = nv.anchor[sl.c];
      s_src[sl.m] = sl.start;
      s_cnt[sl.m] = sl.cnt;
      s_coff[sl.m] = sl.off;
      s_dx[sl.m] = (float)(ab.x - ac.x);
      s_dy[sl.m] = (float)(ab.y - ac.y);
      s_thr[sl.m] = fmaxf(fallback_r2_b<K>(nv.span[b], nv.span[sl.c]), 1.0e-30f);
    }
    if (threadIdx.x == 0) {
      s_coff[sl.ns] = sl.total;
      s_ns = sl.ns;
    }
  }
  __syncthreads();
  const int ns = s_ns;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  double* sacc = (double*)smem + (long)warp * NE * 32;  // lane-major: sum e of lane l at e*32 + l
  float2* sx = (float2*)((double*)smem + (long)nw * NE * 32);
  for (int m = 0; m < ns; ++m) {
    const int o = s_coff[m] * 8, nc = s_cnt[m], src = s_src[m], np = (s_coff[m + 1] - s_coff[m]) * 8;
    const float ddx = s_dx[m], ddy = s_dy[m];
    for (int t = threadIdx.x; t < np; t += blockDim.x) {
      float2 p = make_float2(kPadSrc, kPadSrc);
      if (t < nc) {
        p = nv.rel[src + t];
        p.x -= ddx;
        p.y -= ddy;
      }
      sx[o + t] = p;
    }
  }
  __syncthreads();
  const int gq = lane >> 2, tq = lane & 3;
  for (int tg = warp; tg * 32 < n; tg += nw) {
    // targets of this lane: rows gq, gq + 8 of tile 0 (k = 0, 1) and of tile 1 (k = 2, 3)
    float2 x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int ti = tg * 32 + k * 8 + gq;
      x[k] = ti < n ? nv.rel[s0 + ti] : make_float2(kPadTgt, kPadTgt);
    }
#pragma unroll
    for (int e = 0; e < NE; ++e) sacc[e * 32 + lane] = 0.0;
    for (int m = 0; m < ns; ++m) {
      const int src = s_src[m], nc = s_cnt[m];
      const float thr = s_thr[m];
      float cm[2][RC / 8][4], cc[2][RC / 8][4];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int t = 0; t < RC / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) cm[u][t][e] = cc[u][t][e] = 0.0f;
      for (int c = s_coff[m]; c < s_coff[m + 1]; ++c) {
        const int j0 = (c - s_coff[m]) * 8;
        const float2 ps[2] = {sx[c * 8 + tq], sx[c * 8 + tq + 4]};
        float kv[4][2];
        bool close = false;
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float dx = x[k].x - ps[h].x, dy = x[k].y - ps[h].y;
            const float r2 = fmaf(dx, dx, dy * dy);
            close |= r2 < thr;
            // close pairs (R2 = 0 among them) are overwritten by the FP64 fallback below
            kv[k][h] = K::eval32_pos(r2, a32, p32);
          }
        if (__any_sync(0xffffffffu, close)) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const float dx = x[k].x - ps[h].x, dy = x[k].y - ps[h].y;
              if (fmaf(dx, dx, dy * dy) < thr) {  // both points are real (stand-ins are never close)
                const int pi = s0 + tg * 32 + k * 8 + gq, qi = src + j0 + tq + 4 * h;
                if (pi == qi) {
                  kv[k][h] = (float)K::at_zero(kp);
                } else {
                  const double2 pa = nv.pts[pi], pc = nv.pts[qi];
                  kv[k][h] = (float)K::eval_exact(r2_exact(pa.x, pa.y, pc.x, pc.y), kp);
                }
              }
            }
        }
        // A fragments: tile u rows (gq, gq + 8) = targets 2u, 2u + 1
        uint32_t ah[2][4], al[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          split_tf32_mask(kv[2 * u][0], ah[u][0], al[u][0]);
          split_tf32_mask(kv[2 * u + 1][0], ah[u][1], al[u][1]);
          split_tf32_mask(kv[2 * u][1], ah[u][2], al[u][2]);
          split_tf32_mask(kv[2 * u + 1][1], ah[u][3], al[u][3]);
        }
        const bool va = j0 + tq < nc, vb = j0 + tq + 4 < nc;
        // column tile t of 16 columns takes the columns 2 gq + t: a lane's two charges are neighbours
        const uint2* ra = qhl + (long)(src + j0 + tq) * RC + RC / 8 * gq;
        const uint2* rb = ra + 4 * RC;
        uint2 b0[RC / 8], b1[RC / 8];
        if constexpr (RC == 16) {
          const uint4 w0 = va ? *reinterpret_cast<const uint4*>(ra) : make_uint4(0u, 0u, 0u, 0u);
          const uint4 w1 = vb ? *reinterpret_cast<const uint4*>(rb) : make_uint4(0u, 0u, 0u, 0u);
          b0[0] = make_uint2(w0.x, w0.y);
          b0[1] = make_uint2(w0.z, w0.w);
          b1[0] = make_uint2(w1.x, w1.y);
          b1[1] = make_uint2(w1.z, w1.w);
        } else {
          b0[0] = va ? *ra : make_uint2(0u, 0u);
          b1[0] = vb ? *rb : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int t = 0; t < RC / 8; ++t) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            mma_tf32_16x8x8(cm[u][t], ah[u], b0[t].x, b1[t].x);
            mma_tf32_16x8x8(cc[u][t], ah[u], b0[t].y, b1[t].y);
            mma_tf32_16x8x8(cc[u][t], al[u], b0[t].x, b1[t].x);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int t = 0; t < RC / 8; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            sacc[((u * (RC / 8) + t) * 4 + e) * 32 + lane] += (double)cm[u][t][e] + (double)cc[u][t][e];
    }
    // D fragment of tile u: rows gq (e = 0, 1) and gq + 8 (e = 2, 3), columns RC/4 tq ..: two of a tile,
    // four of two interleaved tiles
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const int ti = tg * 32 + (2 * u + hr) * 8 + gq;
        if (ti < n) {
          double2* o = reinterpret_cast<double2*>(ys + (long)(s0 + ti) * RC + RC / 4 * tq);
          auto sum = [&](int t, int e) { return sacc[((u * (RC / 8) + t) * 4 + 2 * hr + e) * 32 + lane]; };
#pragma unroll
          for (int h = 0; h < RC / 8; ++h) {
            double2 w = o[h];
            w.x += RC == 16 ? sum(0, h) : sum(0, 0);
            w.y += RC == 16 ? sum(1, h) : sum(0, 1);
            o[h] = w;
          }
        }
      }
  }
}

// Stand-in coordinates of padded source slots and absent targets of the FP64
// near field (finite entries for every kernel, never stored).
constexpr double kPadSrc64 = 1.0e100, kPadTgt64 = -1.0e100;

// Near field in FP64 on the FP64 tensor cores (AFMM_PREC_FP64_BATCHED): one
// CTA per leaf, one warp per 32 targets (four 8-row tiles sharing every charge
// fragment).  Source leaves (neighbours 0..7, then the leaf itself) are staged
// in shared memory with their exact coordinates, padded to multiples of 4 with
// far stand-ins; each lane evaluates one FP64 entry per tile and 4-source step
// with the FP64 matvec form K::eval (the diagonal included, as in the FP64
// path), and the 8 x 4 entry tiles multiply the 4 x RC FP64 charge blocks
// (mma.sync m8n8k4, FP64 accumulation).  Of a step's four tiles kAhead have
// their entries before their products, and kCtas (0: the compiler's choice) CTAs
// an SM bound the registers: short formulas gain from four at once (1/r, 8
// columns, 12,000 points in 64 leaves 0.38 -> 0.29 ms, 800,000 in 4,096 2.52 -> 2.42; 16
// columns .41 -> .35, 3.44 -> 3.50), the long table-driven functions from enough
// registers to run into each other by themselves (log, 8 columns, kCtas 0 -> 4: .45 ->
// .36, 4.48 -> 4.46; Gaussian .35 -> .27, 3.56 -> 3.43; Gaussian, 16 columns, 819,200
// points 4.46 -> 4.33; log, 16 columns, worse: 5.27 -> 5.63 at 800,000).
template <class K, int RC>
struct DmmaOrder {
  static constexpr bool kGauss = K::id == AFMM_KERNEL_GAUSSIAN, kTable = kGauss || K::id == AFMM_KERNEL_LOG;
  static constexpr int kAhead = !kTable ? 4 : (kGauss && RC == 16 ? 2 : 1);
  static constexpr int kCtas = kTable && (kGauss || RC == 8) ? 4 : 0;
};

template <class K, int RC>
__global__ void __launch_bounds__(128, DmmaOrder<K, RC>::kCtas) k_p2p_dmma(NearView nv, KernelParams kp, const double* __restrict__ qs,
                                                  double* __restrict__ ys) {
  constexpr int NTT = 4;  // 8-row target tiles per warp
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_src[9], s_cnt[9], s_coff[10], s_ns;
  const long b = nv.leaf0 + blockIdx.x;
  const int n = nv.leaf_cnt[b];
  const int s0 = nv.leaf_start[b];
  if (threadIdx.x < 32) {
    const NearSlots sl = near_slots<4>(nv, b, threadIdx.x);
    if (sl.m >= 0) {
      s_src[sl.m] = sl.start;
      s_cnt[sl.m] = sl.cnt;
      s_coff[sl.m] = sl.off;
    }
    if (threadIdx.x == 0) {
      s_coff[sl.ns] = sl.total;
      s_ns = sl.ns;
    }
  }
  __syncthreads();
  const int ns = s_ns;
  double2* sx = (double2*)smem;
  for (int m = 0; m < ns; ++m) {
    const int o = s_coff[m] * 4, nc = s_cnt[m], src = s_src[m], np = (s_coff[m + 1] - s_coff[m]) * 4;
    for (int t = threadIdx.x; t < np; t += blockDim.x)
      sx[o + t] = t < nc ? nv.pts[src + t] : make_double2(kPadSrc64, kPadSrc64);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int trow = lane >> 2, tsrc = lane & 3;
  for (int tg = warp; tg * 32 < n; tg += nw) {
    double2 x[NTT];
#pragma unroll
    for (int u = 0; u < NTT; ++u) {
      const int ti = tg * 32 + u * 8 + trow;
      x[u] = ti < n ? nv.pts[s0 + ti] : make_double2(kPadTgt64, kPadTgt64);
    }
    double c[NTT][RC / 8][2];
#pragma unroll
    for (int u = 0; u < NTT; ++u)
#pragma unroll
      for (int t = 0; t < RC / 8; ++t) c[u][t][0] = c[u][t][1] = 0.0;
    for (int m = 0; m < ns; ++m) {
      const int src = s_src[m], nc = s_cnt[m];
      for (int st = s_coff[m]; st < s_coff[m + 1]; ++st) {
        const int j = (st - s_coff[m]) * 4 + tsrc;
        const double2 p = sx[st * 4 + tsrc];
        const bool vj = j < nc;
        double bq[RC / 8];
        load_b<RC>(qs + (long)(src + j) * RC, trow, vj, bq);
        constexpr int A = DmmaOrder<K, RC>::kAhead;
#pragma unroll
        for (int u0 = 0; u0 < NTT; u0 += A) {
          double a[A];
#pragma unroll
          for (int u = 0; u < A; ++u) {
            const double dx = x[u0 + u].x - p.x, dy = x[u0 + u].y - p.y;
            a[u] = K::eval(dx * dx + dy * dy, kp);
          }
#pragma unroll
          for (int u = 0; u < A; ++u)
#pragma unroll
            for (int t = 0; t < RC / 8; ++t) mma_f64_8x8x4(c[u0 + u][t][0], c[u0 + u][t][1], a[u], bq[t]);
        }
      }
    }
    // D fragment: row trow, columns RC/4 tsrc .. (load_b's column order)
#pragma unroll
    for (int u = 0; u < NTT; ++u) {
      const int ti = tg * 32 + u * 8 + trow;
      if (ti < n) {
        double2* o = reinterpret_cast<double2*>(ys + (long)(s0 + ti) * RC + RC / 4 * tsrc);
#pragma unroll
        for (int h = 0; h < RC / 8; ++h) {
          double2 w = o[h];
          w.x += RC == 16 ? c[u][0][h] : c[u][0][0];
          w.y += RC == 16 ? c[u][RC / 8 - 1][h] : c[u][0][1];
          o[h] = w;
        }
      }
    }
  }
}

// The FP64 near field of a pass with every unordered pair of leaves worked out
// once (the pairs of near_leaf, fmm.cuh; K(x, y) depends on |x - y| only): one
// CTA per leaf, each warp blocks of 32 points of the leaf's five source leaves
// against all targets, 8 x 8 entries at a time.  An entry is evaluated in the
// lane that holds it in the A fragment of the targets' product (8 targets x 4
// sources); two exchanges between lanes turn it into the A fragment of the sources'
// product (8 sources x 4 targets).  The sources' sums stay in registers over
// all targets, the targets' in a shared-memory row of the warp, added in warp
// order at the end.  part: kNearParts x n x RC.  FP64 datapath: an entry costs
// ~25 operations (log) and RC / 2 in each product, so evaluating it once takes the
// 9 (25 + RC / 2) of a point's row to 5 (25 + RC); it keeps that datapath 61% busy
// (k_p2p_dmma ~69%), with fixed-latency stalls at 15 warps an SM (1,048,576
// points, 16 columns: log 1.94 -> 1.50 ms, Gaussian 1.60 -> 1.37).
template <class K, int RC>
__global__ void __launch_bounds__(256, 2) k_near_dmma(NearView nv, KernelParams kp, const double* __restrict__ qs,
                                                      double* __restrict__ part, int warps) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ NearSources src;
  const long b = nv.run ? (long)nv.run[blockIdx.x] : nv.leaf0 + blockIdx.x;
  const int n = nv.leaf_cnt[b], n8 = (n + 7) & ~7;
  const int s0 = nv.leaf_start[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) src.make(nv, b, lane);
  double2* px = (double2*)smem;                       // targets
  double2* sx = px + n8 + warp * 32;                  // the warp's sources
  double* accs = (double*)(px + n8 + warps * 32);     // the warps' sums of the targets
  double* acc = accs + (size_t)warp * n8 * RC;
  // (targets and sources past the last are the last one again, with no charge: a
  // far-off place would make a growing user kernel's entries overflow, and 0 * inf is not 0)
  for (int i = threadIdx.x; i < n8; i += blockDim.x) px[i] = nv.pts[s0 + min(i, n - 1)];
  for (int i = threadIdx.x; i < warps * n8 * RC; i += blockDim.x) accs[i] = 0.0;
  __syncthreads();
  const int ns = src.ns, total = src.off[ns], nblk = (total + 31) >> 5;
  const int trow = lane >> 2, tsrc = lane & 3;
  const int from = 4 * (tsrc + (trow & 4)) + (trow & 3);
  const int b1 = (warp + 1) * nblk / warps;
  for (int blk = warp * nblk / warps; blk < b1; ++blk) {
    const int f = min(32 * blk + lane, total - 1);
    int m = 0;
    while (m + 1 < ns && f >= src.off[m + 1]) ++m;
    const bool ok = 32 * blk + lane < total;
    const int place = src.src[m] + (f - src.off[m]);
    const int idx = ok ? place : -1;  // the lane's source
    const int dst = ok ? src.dst[m] : 0;
    __syncwarp();
    sx[lane] = nv.pts[place];
    __syncwarp();
    const bool both = __any_sync(0xffffffffu, dst > 0);  // (a block of the leaf's own points: one product)
    double qc[8][RC / 8], yc[4][RC / 8][2];
#pragma unroll
    for (int h = 0; h < 8; ++h) {
      const int j = __shfl_sync(0xffffffffu, idx, 4 * h + tsrc);
      load_b<RC>(qs + (long)max(j, 0) * RC, trow, j >= 0, qc[h]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int t = 0; t < RC / 8; ++t) yc[u][t][0] = yc[u][t][1] = 0.0;
    for (int i0 = 0; i0 < n8; i0 += 8) {
      const double2 xi = px[i0 + trow];
      double qb[2][RC / 8], yb[RC / 8][2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + 4 * h + tsrc;
        load_b<RC>(qs + (long)(s0 + min(i, n - 1)) * RC, trow, i < n, qb[h]);
      }
      double2* o = reinterpret_cast<double2*>(acc + (size_t)(i0 + trow) * RC + RC / 4 * tsrc);
#pragma unroll
      for (int h = 0; h < RC / 8; ++h) {  // (columns in load_b's order)
        const double2 w = o[h];
        if (RC == 16) {
          yb[0][h] = w.x;
          yb[RC / 8 - 1][h] = w.y;
        } else {
          yb[0][0] = w.x;
          yb[0][1] = w.y;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        double e[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double2 p = sx[8 * u + 4 * h + tsrc];
          const double dx = xi.x - p.x, dy = xi.y - p.y;
          e[h] = K::eval(dx * dx + dy * dy, kp);
#pragma unroll
          for (int t = 0; t < RC / 8; ++t) mma_f64_8x8x4(yb[t][0], yb[t][1], e[h], qc[2 * u + h][t]);
        }
        if (both) {
          // entry (i, j), in lane 4 i + (j & 3) and e[j / 4], to lane 4 j + (i & 3) and
          // v[i / 4]: each lane sends and receives one entry twice
          const double x = __shfl_sync(0xffffffffu, trow < 4 ? e[0] : e[1], from);
          const double y = __shfl_sync(0xffffffffu, trow < 4 ? e[1] : e[0], from ^ 16);
          const double v[2] = {trow < 4 ? x : y, trow < 4 ? y : x};
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int t = 0; t < RC / 8; ++t) mma_f64_8x8x4(yc[u][t][0], yc[u][t][1], v[h], qb[h][t]);
        }
      }
#pragma unroll
      for (int h = 0; h < RC / 8; ++h)
        o[h] = RC == 16 ? make_double2(yb[0][h], yb[RC / 8 - 1][h]) : make_double2(yb[0][0], yb[0][1]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = __shfl_sync(0xffffffffu, idx, 8 * u + trow), d = __shfl_sync(0xffffffffu, dst, 8 * u + trow);
      if (d > 0 && d != kNoPart) {
        double2* o = reinterpret_cast<double2*>(part + ((size_t)(d - 1) * nv.n + j) * RC + RC / 4 * tsrc);
#pragma unroll
        for (int h = 0; h < RC / 8; ++h)
          o[h] = RC == 16 ? make_double2(yc[u][0][h], yc[u][RC / 8 - 1][h]) : make_double2(yc[u][0][0], yc[u][0][1]);
      }
    }
  }
  __syncthreads();
  if (b < nv.leaf0 || b >= nv.leaf0 + nv.nleaf) return;
  for (int e = threadIdx.x; e < n * RC; e += blockDim.x) {
    double v = accs[e];
    for (int w = 1; w < warps; ++w) v += accs[(size_t)w * n8 * RC + e];
    part[(size_t)s0 * RC + e] = v;
    for (int s = 0; s < 4; ++s)
      if (!src.back[s]) part[((size_t)(1 + s) * nv.n + s0) * RC + e] = 0.0;
  }
}

inline int nbk(long n, int t) { return (int)((n + t - 1) / t); }

// M2L with the entries evaluated on the fly, RC = 8 or 16 columns per pass,
// on FP64 tensor-core tiles (k_m2l_mma).
template <class K, int RC>
void m2l_otf_batched(const LevelSet& ls, const KernelParams& kp, const double* const* qh, double* const* yh,
                     cudaStream_t s) {
  if (ls.row0[ls.nlev] == 0) return;
  const long warps = ls.grp0[ls.nlev];
  k_m2l_mma<K, RC><<<nbk(warps * 32, 128), 128, 0, s>>>(ls, kp, qh, yh);
  AFMM_LAUNCH_CHECK();
}

// Mixed near field of a pass: TF32x3 tensor-core tiles (8 or 16 columns,
// charges as TF32 parts).
template <class K, int RC>
void p2p_mma_batched(const NearView& nv, const KernelParams& kp, const uint2* qhl, double* ys, cudaStream_t s) {
  const int warps = std::min(4, (nv.nmax + 31) / 32);
  const size_t smem = (size_t)9 * ((nv.nmax + 7) / 8 * 8) * sizeof(float2) + (size_t)warps * RC * 32 * sizeof(double);
  allow_smem(k_p2p_mma<K, RC>, smem);
  k_p2p_mma<K, RC><<<(int)nv.nleaf, 32 * warps, smem, s>>>(nv, kp, qhl, ys);
  AFMM_LAUNCH_CHECK();
}

template <int RC>
size_t near_dmma_smem(int nmax, int warps) {
  const size_t n8 = (nmax + 7) & ~7;
  return (n8 + 32 * warps) * sizeof(double2) + (size_t)warps * n8 * RC * sizeof(double);
}

// Its warps: four or five, whichever share the blocks more evenly (an SM holds
// 16 of the kernel's warps: smaller CTAs leave less of it idle at the end of each);
// near_warps's up to eight when the leaves are few.
inline int near_dmma_warps(int nmax, bool few) {
  if (few) return near_warps(nmax);
  const int blocks = (5 * nmax + 31) / 32;
  if (blocks <= 5) return std::max(blocks, 1);
  return 5 * ((blocks + 4) / 5) <= 4 * ((blocks + 3) / 4) ? 5 : 4;
}

// k_near_dmma for all leaves of nv, when it is the better form (false: k_p2p_dmma).
// The line, in FP64 operations per point at 16 columns: k_p2p_dmma works out
// nine leaves of points in groups of 32 targets, a warp each, up to four warps a
// CTA, so that with five or six groups warps wait in the second round (`idle`);
// k_near_dmma works out five in groups of 8 and moves 1 KB of parts (~2,500
// operations' time), and with fewer than three CTAs an SM its latencies show.
// Whole calls, 16 columns, k_p2p_dmma / k_near_dmma, log, Gaussian, scaled 1/r, 1/r
// (ms; 4,096 leaves, above 16,384):
//   leaves of 48 points  2.19 / 1.70  1.72 / 1.43  2.03 / 1.81  1.83 / 1.70
//             56         2.47 / 2.13  1.94 / 1.81  2.26 / 2.20  2.03 / 2.06
//             88         1.39 / 1.10  1.17 / 1.01  1.15 / 1.06  1.04 / 0.99
//             112        2.00 / 1.85  1.64 / 1.66  1.63 / 1.66  1.47 / 1.62
//             136        3.23 / 2.34  2.63 / 2.12  2.58 / 2.00  2.47 / 1.93
//             152        3.63 / 3.09  2.97 / 2.83  2.93 / 2.68  2.84 / 2.62
//             200        5.83 / 5.24  4.81 / 4.79  4.51 / 4.33  3.97 / 4.26
// and with 32-point leaves (524,288 points) 1.16 / 1.14, .88 / .94, 1.21 / 1.28,
// 1.13 / 1.22.  With too few leaves to fill the GPU (`few`: up to two an SM) what
// counts is that five to eight warps share a leaf instead of one per 32 targets
// (4,096 points, 91 -> 41 us; 12,000 points in 64 leaves .44 -> .17 ms), whatever shared
// memory their target rows take.
template <class K, int RC>
bool near_dmma_batched(const NearView& nv, const KernelParams& kp, const double* qs, double* part, bool launch,
                       cudaStream_t s) {
  const bool few = nv.n <= 2L * sm_count() * nv.nmax;
  const int warps = near_dmma_warps(nv.nmax, few);
  const size_t smem16 = near_dmma_smem<16>(nv.nmax, warps);
  if (smem16 > (few ? 220 : 110) * 1024) return false;
  constexpr double entry = K::id == AFMM_KERNEL_LOG                ? 25.0
                           : K::id == AFMM_KERNEL_GAUSSIAN         ? 16.0
                           : K::id == AFMM_KERNEL_ONE_OVER_R_SCALED ? 13.0
                                                                    : 8.0;
  const int groups = (nv.nmax + 31) / 32;
  const double idle = groups > 4 ? 1.0 - groups / (4.0 * ((groups + 3) / 4)) : 0.0;
  const double twice = 9.0 * (32 * groups) * (entry + 8.0) * (1.0 + 1.8 * idle * idle);
  const double once = (5.0 * ((nv.nmax + 7) & ~7) * (entry + 16.0) + 2500.0) * (smem16 > 74 * 1024 ? 1.29 : 1.0);
  if (!few && 1.05 * once > twice) return false;
  if (!launch) return true;
  const size_t smem = near_dmma_smem<RC>(nv.nmax, warps);
  allow_smem(k_near_dmma<K, RC>, smem);
  k_near_dmma<K, RC><<<(int)(nv.run ? nv.nrun : nv.nleaf), 32 * warps, smem, s>>>(nv, kp, qs, part, warps);
  AFMM_LAUNCH_CHECK();
  return true;
}

// FP64 near field of an FP64-batched pass (8 or 16 columns).
template <class K, int RC>
void p2p_dmma_batched(const NearView& nv, const KernelParams& kp, const double* qs, double* ys, cudaStream_t s) {
  const int warps = std::min(4, (nv.nmax + 31) / 32);
  const size_t smem = (size_t)9 * ((nv.nmax + 3) / 4 * 4) * sizeof(double2);
  allow_smem(k_p2p_dmma<K, RC>, smem);
  k_p2p_dmma<K, RC><<<(int)nv.nleaf, 32 * warps, smem, s>>>(nv, kp, qs, ys);
  AFMM_LAUNCH_CHECK();
}

}  // namespace batched_detail

}  // namespace afmm
