// More user kernels defined outside the library: the polyharmonic spline
// K(r) = r^4 log r, which grows with the distance, and exp(-r^2 / c), whose
// matvec entries call the library's FP64 logarithm and exponential by the
// names first offered to user kernels; and cos(c r), of full rank when its waves
// are shorter than the points' distances.
#include "afmm2d_kernel.cuh"

struct PolyharmonicSpline {
  static constexpr int id = AFMM_KERNEL_USER_FIRST + 8;
  __device__ __forceinline__ static double at_zero(const afmm::KernelParams&) { return 0.0; }
  __device__ __forceinline__ static double eval_exact(double R2, const afmm::KernelParams&) {
    return R2 == 0.0 ? 0.0 : __dmul_rn(__dmul_rn(__dmul_rn(0.5, R2), R2), afmm::log_cr(R2));
  }
  __device__ __forceinline__ static double eval(double R2, const afmm::KernelParams&) {
    return R2 == 0.0 ? 0.0 : 0.5 * R2 * R2 * afmm::log_tang(R2);
  }
  __device__ __forceinline__ static float eval32(float R2, float, float) {
    return R2 == 0.0f ? 0.0f : 0.5f * R2 * R2 * logf(R2);
  }
  __device__ __forceinline__ static float eval32_pos(float R2, float a, float c) { return eval32(R2, a, c); }
};

struct UserGaussian {
  static constexpr int id = AFMM_KERNEL_USER_FIRST + 9;
  __device__ __forceinline__ static double at_zero(const afmm::KernelParams&) { return 1.0; }
  __device__ __forceinline__ static double eval_exact(double R2, const afmm::KernelParams& p) {
    return afmm::exp_cr(-__ddiv_rn(R2, p.param));
  }
  __device__ __forceinline__ static double eval(double R2, const afmm::KernelParams& p) {
    return afmm::exp_tang(-R2 / p.param);
  }
  __device__ __forceinline__ static float eval32(float R2, float, float c) { return expf(-R2 / c); }
  __device__ __forceinline__ static float eval32_pos(float R2, float a, float c) { return eval32(R2, a, c); }
};

struct Wave {
  static constexpr int id = AFMM_KERNEL_USER_FIRST + 10;
  __device__ __forceinline__ static double at_zero(const afmm::KernelParams&) { return 1.0; }
  __device__ __forceinline__ static double eval_exact(double R2, const afmm::KernelParams& p) {
    return cos(__dmul_rn(p.param, __dsqrt_rn(R2)));
  }
  __device__ __forceinline__ static double eval(double R2, const afmm::KernelParams& p) { return eval_exact(R2, p); }
  __device__ __forceinline__ static float eval32(float R2, float, float c) { return cosf(c * sqrtf(R2)); }
  __device__ __forceinline__ static float eval32_pos(float R2, float a, float c) { return eval32(R2, a, c); }
};

AFMM_REGISTER_KERNEL(PolyharmonicSpline)
AFMM_REGISTER_KERNEL(UserGaussian)
AFMM_REGISTER_KERNEL(Wave)
