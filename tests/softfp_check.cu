// The Soft arithmetic (csrc/softfp.cuh) over arrays: on the GPU
// when compiled by nvcc, else on the host with a stand-in for the MUFU seeds
// (off by `rel`, to cover the bounds of MUFU's error).
#include "softfp.cuh"

using namespace amr;

AMR_HD void check_one(double a, double b, double *q, double *r, double *q3, double *q6, unsigned char *bad) {
  bool f = false, g = false, h = false, k = false;
  *q = div_rn(a, b, f);
  *r = sqrt_rn(a, g);
  *q3 = div_by<3>(a, h);
  *q6 = div_by<6>(a, k);
  *bad = static_cast<unsigned char>(f | g << 1 | h << 2 | k << 3);
}

// product, double to float and back
AMR_HD void check_mul(double a, double b, double *p, double *f, double *d, unsigned char *bad) {
  bool g = false;
  *p = mul_rn(a, b, g);
  const float x = to_f32(a);
  *f = x;
  *d = to_f64(x);
  *bad = static_cast<unsigned char>(g);
}

#ifdef __CUDACC__
__global__ void k_mul(const double *a, const double *b, long n, double *o, unsigned char *bad) {
  const long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) check_mul(a[i], b[i], o + i, o + n + i, o + 2 * n + i, bad + i);
}
extern "C" int softmul_check(const double *a, const double *b, long n, double *out, unsigned char *bad) {
  double *d = nullptr;
  unsigned char *e = nullptr;
  cudaError_t rc = cudaMalloc(&d, 5 * n * sizeof(double));
  if (rc == cudaSuccess) rc = cudaMalloc(&e, n);
  if (rc == cudaSuccess) rc = cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
  if (rc == cudaSuccess) rc = cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
  if (rc == cudaSuccess) {
    k_mul<<<static_cast<unsigned>((n + 255) / 256), 256>>>(d, d + n, n, d + 2 * n, e);
    rc = cudaGetLastError();
  }
  if (rc == cudaSuccess) rc = cudaMemcpy(out, d + 2 * n, 3 * n * sizeof(double), cudaMemcpyDeviceToHost);
  if (rc == cudaSuccess) rc = cudaMemcpy(bad, e, n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(e);
  return static_cast<int>(rc);
}
#else
extern "C" int softmul_check(const double *a, const double *b, long n, double *out, unsigned char *bad) {
  for (long i = 0; i < n; i++) check_mul(a[i], b[i], out + i, out + n + i, out + 2 * n + i, bad + i);
  return 0;
}
#endif

#ifdef __CUDACC__
__global__ void k_check(const double *a, const double *b, long n, double *o, unsigned char *bad) {
  const long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) check_one(a[i], b[i], o + i, o + n + i, o + 2 * n + i, o + 3 * n + i, bad + i);
}
extern "C" int softfp_check(const double *a, const double *b, long n, double, double *out, unsigned char *bad) {
  double *d = nullptr;
  unsigned char *e = nullptr;
  cudaError_t rc = cudaMalloc(&d, 6 * n * sizeof(double));
  if (rc == cudaSuccess) rc = cudaMalloc(&e, n);
  if (rc == cudaSuccess) rc = cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
  if (rc == cudaSuccess) rc = cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
  if (rc == cudaSuccess) {
    k_check<<<static_cast<unsigned>((n + 255) / 256), 256>>>(d, d + n, n, d + 2 * n, e);
    rc = cudaGetLastError();
  }
  if (rc == cudaSuccess) rc = cudaMemcpy(out, d + 2 * n, 4 * n * sizeof(double), cudaMemcpyDeviceToHost);
  if (rc == cudaSuccess) rc = cudaMemcpy(bad, e, n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(e);
  return static_cast<int>(rc);
}
#else
extern "C" int softfp_check(const double *a, const double *b, long n, double rel, double *out, unsigned char *bad) {
  seed_rel() = rel;
  for (long i = 0; i < n; i++) check_one(a[i], b[i], out + i, out + n + i, out + 2 * n + i, out + 3 * n + i, bad + i);
  return 0;
}
#endif
