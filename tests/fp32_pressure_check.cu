// The FP32 path's pressure recovery (cons2prim_cell<float>, csrc/stage.cuh) over
// an array of conserved states, and the same pairs of floats summed in FP64.
#include "stage.cuh"

using namespace amr;

__device__ float summed_in_fp64(const float *u, double g) {
  const float ir = 1.0f / u[0];
  const float rl = __fmul_rn(__fmaf_rn(-u[0], ir, 1.0f), ir);
  float mh, ml, bh, bl;
  sum_sq3(u[1], u[2], u[3], mh, ml);
  sum_sq3(u[5], u[6], u[7], bh, bl);
  const float kh = __fmul_rn(mh, ir);
  const float kl = __fadd_rn(__fmaf_rn(mh, ir, -kh), __fadd_rn(__fmul_rn(mh, rl), __fmul_rn(ml, ir)));
  const double b2 = static_cast<double>(bh) + static_cast<double>(bl);
  return static_cast<float>((g - 1) * (u[4] - 0.5 * ((static_cast<double>(kh) + static_cast<double>(kl)) + b2)));
}

__global__ void k_pressure(const float *u, long n, double gamma, float *p, float *q) {
  const long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float v[8], w[8];
  for (int k = 0; k < 8; k++) v[k] = u[8 * i + k];
  InstParams ip{};
  ip.gm1_hi = static_cast<float>(gamma - 1);
  ip.gm1_lo = static_cast<float>((gamma - 1) - static_cast<double>(ip.gm1_hi));
  cons2prim_cell<float>(v, w, GasGamma<float>(ip));
  p[i] = w[4];
  q[i] = summed_in_fp64(v, gamma);
}

extern "C" int fp32_pressure(const float *u, long n, double gamma, float *p, float *q) {
  float *d = nullptr;
  cudaError_t rc = cudaMalloc(&d, 10 * n * sizeof(float));
  if (rc != cudaSuccess) return static_cast<int>(rc);
  rc = cudaMemcpy(d, u, 8 * n * sizeof(float), cudaMemcpyHostToDevice);
  if (rc == cudaSuccess) {
    k_pressure<<<static_cast<unsigned>((n + 255) / 256), 256>>>(d, n, gamma, d + 8 * n, d + 9 * n);
    rc = cudaGetLastError();
  }
  if (rc == cudaSuccess) rc = cudaMemcpy(p, d + 8 * n, n * sizeof(float), cudaMemcpyDeviceToHost);
  if (rc == cudaSuccess) rc = cudaMemcpy(q, d + 9 * n, n * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return static_cast<int>(rc);
}
