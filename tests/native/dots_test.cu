// The ACA's dot-product accumulation (dd_add_product, aca_k.cuh): the terms of
// the file (n, then n x's and n y's, doubles) added up by one thread in order;
// prints the pair's two words.  Needs a GPU.
#include <cstdio>
#include <vector>

#include "../../afmm2d_b200/csrc/aca_k.cuh"

__global__ void k_dot(const double* x, const double* y, int n, double* out) {
  afmm::dd a{0.0, 0.0};
  for (int i = 0; i < n; ++i) afmm::aca_detail::dd_add_product(a, x[i], y[i]);
  out[0] = a.hi;
  out[1] = a.lo;
}

int main(int argc, char** argv) {
  FILE* f = argc > 1 ? std::fopen(argv[1], "rb") : nullptr;
  double dn = 0;
  if (!f || std::fread(&dn, 8, 1, f) != 1 || !(dn >= 1 && dn < 1e6)) return 2;
  const int n = (int)dn;
  std::vector<double> v(2 * (size_t)n);
  if (std::fread(v.data(), 8, v.size(), f) != v.size()) return 2;
  std::fclose(f);
  double *d = nullptr, *out = nullptr, r[2];
  if (cudaMalloc(&d, 8 * v.size()) || cudaMalloc(&out, 16)) return 3;
  if (cudaMemcpy(d, v.data(), 8 * v.size(), cudaMemcpyHostToDevice)) return 3;
  k_dot<<<1, 1>>>(d, d + n, n, out);
  if (cudaMemcpy(r, out, 16, cudaMemcpyDeviceToHost)) return 3;
  std::printf("%a %a\n", r[0], r[1]);
  return 0;
}
