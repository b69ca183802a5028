// The Soft arithmetic's products with powers of two (csrc/softfp.cuh) over
// arrays: on the GPU when compiled by nvcc, else on the host.  out: x/4, x/2, 2x,
// 4x, x p; bad: one bit each.
#include "softfp.cuh"

using namespace amr;

AMR_HD void check_one(double x, double p, double *o, long n, unsigned char *bad) {
  bool b[5] = {false, false, false, false, false};
  o[0] = scale_pow2<-2>(x, b[0]);
  o[n] = scale_pow2<-1>(x, b[1]);
  o[2 * n] = scale_pow2<1>(x, b[2]);
  o[3 * n] = scale_pow2<2>(x, b[3]);
  o[4 * n] = times_pow2(x, p, b[4]);
  *bad = static_cast<unsigned char>(b[0] | b[1] << 1 | b[2] << 2 | b[3] << 3 | b[4] << 4);
}

#ifdef __CUDACC__
__global__ void k_check(const double *x, const double *p, long n, double *o, unsigned char *bad) {
  const long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) check_one(x[i], p[i], o + i, n, bad + i);
}
extern "C" int pow2_check(const double *x, const double *p, long n, double *out, unsigned char *bad) {
  double *d = nullptr;
  unsigned char *e = nullptr;
  cudaError_t rc = cudaMalloc(&d, 7 * n * sizeof(double));
  if (rc == cudaSuccess) rc = cudaMalloc(&e, n);
  if (rc == cudaSuccess) rc = cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
  if (rc == cudaSuccess) rc = cudaMemcpy(d + n, p, n * sizeof(double), cudaMemcpyHostToDevice);
  if (rc == cudaSuccess) {
    k_check<<<static_cast<unsigned>((n + 255) / 256), 256>>>(d, d + n, n, d + 2 * n, e);
    rc = cudaGetLastError();
  }
  if (rc == cudaSuccess) rc = cudaMemcpy(out, d + 2 * n, 5 * n * sizeof(double), cudaMemcpyDeviceToHost);
  if (rc == cudaSuccess) rc = cudaMemcpy(bad, e, n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(e);
  return static_cast<int>(rc);
}
#else
extern "C" int pow2_check(const double *x, const double *p, long n, double *out, unsigned char *bad) {
  for (long i = 0; i < n; i++) check_one(x[i], p[i], out + i, n, bad + i);
  return 0;
}
#endif
