// Device-function probe for tests/test_phase_fp64.py: the library's FP64
// psi * exp(z) and the short series under it (common.cuh) on exponents read
// from a file.
#include <cstdio>
#include <vector>

#include "common.cuh"

__global__ void probe(const double2 *z, double2 *mul, double2 *cis, double2 *em1, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  mul[i] = dftgpu::mul_cexp(make_double2(0.6, -0.8), z[i]);
  cis[i] = dftgpu::cism1_8th(z[i].y);
  em1[i] = make_double2(dftgpu::expm1_8th(z[i].x), 0.0);
}

int main(int argc, char **argv) {
  if (argc != 3) { fprintf(stderr, "usage: phase_probe_fp64 in.bin out.bin\n"); return 2; }
  FILE *f = fopen(argv[1], "rb");
  if (!f) return 3;
  std::vector<double2> z;
  double2 v;
  while (fread(&v, sizeof(v), 1, f) == 1) z.push_back(v);
  fclose(f);
  const int n = (int) z.size();
  double2 *dz, *out;
  if (cudaMalloc(&dz, n * sizeof(double2)) || cudaMalloc(&out, 3 * (size_t) n * sizeof(double2))) return 4;
  cudaMemcpy(dz, z.data(), n * sizeof(double2), cudaMemcpyHostToDevice);
  probe<<<(n + 255) / 256, 256>>>(dz, out, out + n, out + 2 * (size_t) n, n);
  std::vector<double2> r(3 * (size_t) n);
  if (cudaMemcpy(r.data(), out, r.size() * sizeof(double2), cudaMemcpyDeviceToHost)) return 5;
  FILE *o = fopen(argv[2], "wb");
  if (!o) return 6;
  fwrite(r.data(), sizeof(double2), r.size(), o);
  fclose(o);
  return 0;
}
