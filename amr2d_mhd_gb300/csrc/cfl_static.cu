// amr_cfl_dt_static: the CFL reduction (main.cpp:209-230) for callers that may
// not allocate device memory.
//
// Some hosts cannot call cudaMalloc at the point where they need the time step:
// code running inside a captured CUDA graph, allocator-free real-time loops,
// or frameworks that own every device allocation and forbid others.  This
// entry point takes the caller's device arrays and keeps its only scratch, the
// running minimum and two counts, in this file's device globals, so it
// allocates nothing.
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

#include "../../include/amr2d_mhd.h"
#include "stage.cuh"

namespace amr {

constexpr int kCflStaticMaxBlocks = 1 << 16;

// The minimum over the blocks so far, as a key whose unsigned order is the
// order of the values, the number of NaN blocks and of finished CTAs; shared
// by every call.  The last CTA of a launch writes the result and puts the
// start values back, so a call needs no other launch.
constexpr unsigned long long kCflKeyMax = ~0ull;
static __device__ unsigned long long g_cfl_key = kCflKeyMax;
static __device__ unsigned g_cfl_nans = 0, g_cfl_done = 0;

__device__ __forceinline__ unsigned long long cfl_key(double v) {
  const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
  return u >> 63 ? ~u : u | (1ull << 63);
}
__device__ __forceinline__ double cfl_unkey(unsigned long long k) {
  return __longlong_as_double(static_cast<long long>(k >> 63 ? k & ~(1ull << 63) : ~k));
}

// Bound by the FP64 pipe: about 35 FP64 instructions per cell, the divisions
// and square roots on the integer pipe (softfp.cuh), and the maximum, where a
// NaN counts as the largest, on the bit patterns.  One thread per interior
// cell; the minimum over the blocks by an atomic of each CTA, taken over by
// the last one.  20011 blocks: 0.37 ms (0.72 with a
// loop over all cells of a block and a second launch for the minimum, 2.25 at
// first), 64 blocks 9 us (18, 29).
//
// main.cpp:211-228 for one block of the dense array: lambda1 takes |rho| +
// c_f,x (W[..][0], main.cpp:222) and lambda2 |u| + c_f,y (:224) over the
// interior cells; lambda = min(1e6, min over blocks) (main.cpp:209,228); a
// NaN block value makes the result NaN, which the caller's invalid-dt check
// catches
template <int NG>
__global__ void __launch_bounds__(256) k_cfl_static(const double *U, const double *dxdy, double gamma, double *out) {
  constexpr int N = Geo<NG>::N, NN = N * N;
  static_assert(NI * NI == 256, "one thread per interior cell");
  __shared__ unsigned long long red[8];
  const double *u0 = U + static_cast<size_t>(blockIdx.x) * 8 * NN;
  const int c = (NG + threadIdx.x / NI) * N + NG + threadIdx.x % NI;
  double u[8], w[8];
#pragma unroll
  for (int k = 0; k < 8; k++) u[k] = u0[k * NN + c];
  cons2prim_cell<double>(u, w, GasGamma<double>(gamma));
  double v1 = 0, v2 = 0;
  evaluate<double>([&](auto &ar) {
    double cf[2];
    fast_speeds<double>(ar, w, gamma, cf);
    v1 = fabs(w[0]) + cf[0];
    v2 = fabs(w[1]) + cf[1];
  });
  // neither speed is negative: their bits are in their order, a NaN (its sign
  // taken off) above all
  auto bits = [](double v) {
    return bits_nan(v) ? 0x7ff8000000000000ull : static_cast<unsigned long long>(__double_as_longlong(v));
  };
  const unsigned long long b1 = bits(v1), b2 = bits(v2);
  unsigned long long m = b1 > b2 ? b1 : b2;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
    m = v > m ? v : m;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int q = 1; q < 8; q++) m = red[q] > m ? red[q] : m;
  const double v = smin(dxdy[2 * blockIdx.x], dxdy[2 * blockIdx.x + 1]) / __longlong_as_double(static_cast<long long>(m));
  if (isnan(v)) atomicAdd(&g_cfl_nans, 1u);
  else atomicMin(&g_cfl_key, cfl_key(v));
  __threadfence();
  if (atomicAdd(&g_cfl_done, 1u) != gridDim.x - 1) return;
  __threadfence();
  const unsigned nans = atomicExch(&g_cfl_nans, 0u);
  const unsigned long long key = atomicExch(&g_cfl_key, kCflKeyMax);
  g_cfl_done = 0;
  const double lambda = cfl_unkey(key);
  *out = nans ? NAN : (key != kCflKeyMax && lambda < 1.E6 ? lambda : 1.E6);
}

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_mu;
bool g_loaded[kMaxDevices] = {false};

// Every kernel of this entry point loaded on the current device, once: under
// lazy module loading a kernel first launched inside a stream capture would
// load there.
cudaError_t load_on_current_device() {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_loaded[dev]) {
    cudaFuncAttributes fa;
    if ((e = cudaFuncGetAttributes(&fa, k_cfl_static<2>)) != cudaSuccess) return e;
    if ((e = cudaFuncGetAttributes(&fa, k_cfl_static<4>)) != cudaSuccess) return e;
    g_loaded[dev] = true;
  }
  return cudaSuccess;
}
}  // namespace

}  // namespace amr

extern "C" int amr_cfl_dt_static(const double *U, int32_t nblocks, int32_t nghosts, const double *dxdy,
                                 double gamma, double *dt_per_cfl_out, void *stream) {
  using namespace amr;
  if (!U || !dxdy || !dt_per_cfl_out || nblocks <= 0) return AMR_E_ARG;
  if (nblocks > kCflStaticMaxBlocks) return AMR_E_TOO_LARGE;
  if (nghosts != 2 && nghosts != 4) return AMR_E_CONFIG;
  // an error the caller's own earlier work left pending is theirs: report
  // it without clearing it, and launch nothing
  if (cudaPeekAtLastError() != cudaSuccess) return AMR_E_CUDA;
  if (load_on_current_device() != cudaSuccess) return AMR_E_CUDA;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (nghosts == 2) k_cfl_static<2><<<nblocks, 256, 0, s>>>(U, dxdy, gamma, dt_per_cfl_out);
  else k_cfl_static<4><<<nblocks, 256, 0, s>>>(U, dxdy, gamma, dt_per_cfl_out);
  return cudaGetLastError() == cudaSuccess ? AMR_OK : AMR_E_CUDA;
}
