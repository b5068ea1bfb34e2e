// The library's reciprocals beside CUDA's division and square root, for tests/test_rcp_gpu.py.
#include "rcp.cuh"

static __global__ void k_probe(const double *x, long long n, double *r, double *rs, double *d, double *ds) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = cb2::recip(x[i]);
  rs[i] = cb2::recip_sqrt(fabs(x[i]));
  d[i] = 1.0 / x[i];
  ds[i] = 1.0 / sqrt(fabs(x[i]));
}

extern "C" int probe(const double *x, long long n, double *r, double *rs, double *d, double *ds) {
  k_probe<<<(unsigned)((n + 255) / 256), 256>>>(x, n, r, rs, d, ds);
  return (int)cudaDeviceSynchronize();
}
