// amr_cfl_dt_static: the CFL reduction (main.cpp:209-230) for callers that may
// not allocate device memory.
//
// Some hosts cannot call cudaMalloc at the point where they need the time step:
// code running inside a captured CUDA graph, allocator-free real-time loops,
// or frameworks that own every device allocation and forbid others.  This
// entry point takes the caller's device arrays and has no scratch: it allocates
// nothing.
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

#include "../../include/amr2d_mhd.h"
#include "launch.hpp"
#include "stage.cuh"

namespace amr {

constexpr int kCflStaticMaxBlocks = 1 << 16;

// The result itself is the running minimum, started at the cap by a launch of
// its own, so a call depends on nothing that another call has left and calls
// with results of their own may overlap.
__global__ void k_cfl_start(double *out) {
  asm volatile("griddepcontrol.launch_dependents;");   // k_cfl_static waits for this grid before it looks at *out
  *out = 1.E6;
}

// *out = min(*out, v), and a NaN for good once v is one.  As bit patterns the
// values that are not negative order as signed integers, below them the
// negative ones in reverse as unsigned integers; the NaN taken, all ones, is
// above every negative value in that second order.
__device__ __forceinline__ void cfl_take(double *out, double v) {
  const long long now = *reinterpret_cast<volatile long long *>(out);
  const long long s = isnan(v) ? -1ll : __double_as_longlong(v);
  if (s >= 0) {
    if (s < now) atomicMin(reinterpret_cast<long long *>(out), s);
  } else if (static_cast<unsigned long long>(s) > static_cast<unsigned long long>(now)) {
    atomicMax(reinterpret_cast<unsigned long long *>(out), static_cast<unsigned long long>(s));
  }
}

// Bound by the FP64 pipe: about 35 FP64 instructions per cell, the divisions
// and square roots on the integer pipe (softfp.cuh), and the maximum, where a
// NaN counts as the largest, on the bit patterns.  One thread per interior
// cell; the minimum over the blocks by an atomic of each CTA that lowers it.
// 64 blocks 8.2 us a call, 20011 blocks 370 us.  k_cfl_start beside it costs
// nothing that shows, as a programmatic dependent is launched while its
// predecessor runs (the minimum kept in device globals that the last CTA put
// back, with no second launch: 8.3 and 373 us; the start value by a memset: 9.1
// and 373).
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
  pdl_wait();
  cfl_take(out, v);
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
    if ((e = cudaFuncGetAttributes(&fa, k_cfl_start)) != cudaSuccess) return e;
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
  k_cfl_start<<<1, 1, 0, s>>>(dt_per_cfl_out);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = launch_k(1, nghosts == 2 ? k_cfl_static<2> : k_cfl_static<4>, nblocks, 256, 0, s, U, dxdy, gamma,
                 dt_per_cfl_out);
  if (e == cudaSuccess) return AMR_OK;
  cudaGetLastError();
  return AMR_E_CUDA;
}
