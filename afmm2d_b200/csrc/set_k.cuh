// Kernel-templated stage of many-problem sets: the fused FP64 near field,
// instantiated once per kernel functor by the kernel tables
// (kernel_table.cuh).
#pragma once
#include "set.cuh"

namespace afmm {

namespace set_detail {

// Near field: one CTA per leaf of every problem, each problem with the number
// of warps of its own launch, so the warps' sums add in the same order.
template <class K>
__global__ void __launch_bounds__(256, 3) k_set_p2p64(SetDev d, SetSegs sg) {
  extern __shared__ __align__(16) unsigned char smem[];
  const long g = blockIdx.x;
  const int s = seg_of(sg, g);
  const int p = sg.prob[s];
  const NearView nv = d.nv[p];
  const KernelParams kp = d.kp[p];
  near_leaf<K>(nv, kp, d.qs[p], d.p2p_warps[p], g - sg.first[s], smem);
}

template <class K>
struct SetP2pRun {
  static void prepare(size_t smem) { allow_smem(k_set_p2p64<K>, smem); }
  static void run(const SetPlan& sp, cudaStream_t s) {
    k_set_p2p64<K><<<(int)sp.p2p.total, sp.p2p_threads, sp.p2p_smem, s>>>(sp.dev, sp.p2p);
    AFMM_LAUNCH_CHECK();
  }
};

}  // namespace set_detail

}  // namespace afmm
