// The RK stage as three kernels: primitive variables, Riemann fluxes, and the
// residual + RK update.  Same arithmetic as the fused k_stage (stage.cuh); the
// face kernel spreads the FP64-bound flux work of all leaves evenly over the
// SMs (one thread per face) instead of one CTA per block, and the primitive
// state and fluxes travel through L2 (the whole working set of a step is well
// below the 129 MB L2).
#pragma once

#include "stage.cuh"

namespace amr {

struct SplitArgs {
  const LeafTask *tasks;
  const InstParams *inst;
  const void *qin;    // U (stage 1) or Us (stage 2)
  void *qout;         // Us (stage 1) or U (stage 2)
  void *W;            // primitive state pool [slot][8][N][N]
  const double *B;    // Bi (stage 1) or Bis (stage 2)
  void *ff;
  void *gg;
  DevError *err;
  unsigned *ctr;      // [2] work counter and finished-CTA counter of k_faces_dyn (zero between launches)
  int step;
  int ntasks;
  FillFuse fuse;      // fused fills: the qin fill gathered by k_prim_task, the
                      // flux fill's snapshots saved by k_resid
};

// U2W / Us2W (meshblock.cpp:119-179) for every cell of every leaf
template <int NG, typename S>
__global__ void __launch_bounds__(512) k_prim(SplitArgs a) {
  pdl_wait();
  using G = Geo<NG>;
  constexpr int N = G::N, NN = G::NN, LO = G::LO, HI = G::HI;
  const size_t e = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= static_cast<size_t>(a.ntasks) * NN) return;
  const int t = static_cast<int>(e / NN), c = static_cast<int>(e % NN);
  const LeafTask task = a.tasks[t];
  const size_t base = static_cast<size_t>(task.slot) * 8 * NN;
  const S *Q = static_cast<const S *>(a.qin) + base;
  S *W = static_cast<S *>(a.W) + base;
  S u[8], w[8];
#pragma unroll
  for (int k = 0; k < 8; k++) u[k] = Q[k * NN + c];
  cons2prim_cell<S>(u, w, GasGamma<S>(a.inst[task.inst]));
#pragma unroll
  for (int k = 0; k < 8; k++) W[k * NN + c] = w[k];
  const int i = c % N, j = c / N;
  if (w[4] <= S(0) && i > LO && i < HI + 1 && j > LO && j < HI + 1)
    dev_fail(a.err, DERR_PRESSURE, task.slot, i, j, static_cast<double>(w[4]));
  bool bad = false;
#pragma unroll
  for (int k = 0; k < 8; k++) bad |= bits_nan(w[k]);
  if (bad) dev_fail(a.err, DERR_NAN, task.slot, i, j, 0.0);
}

// the same with the fill of qin (and B) fused in: one CTA per leaf gathers
// its block's ghost cells, then converts the block
template <int NG, typename S>
__global__ void __launch_bounds__(512) k_prim_task(SplitArgs a) {
  pdl_wait();
  using G = Geo<NG>;
  constexpr int N = G::N, NN = G::NN, LO = G::LO, HI = G::HI;
  const LeafTask task = a.tasks[blockIdx.x];
  fill_apply_task<N, S>(a.fuse, task, threadIdx.x, blockDim.x);
  __syncthreads();
  const size_t base = static_cast<size_t>(task.slot) * 8 * NN;
  const S *Q = static_cast<const S *>(a.qin) + base;
  S *W = static_cast<S *>(a.W) + base;
  const GasGamma<S> gamma(a.inst[task.inst]);
  for (int c = threadIdx.x; c < NN; c += blockDim.x) {
    S u[8], w[8];
#pragma unroll
    for (int k = 0; k < 8; k++) u[k] = Q[k * NN + c];
    cons2prim_cell<S>(u, w, gamma);
#pragma unroll
    for (int k = 0; k < 8; k++) W[k * NN + c] = w[k];
    const int i = c % N, j = c / N;
    if (w[4] <= S(0) && i > LO && i < HI + 1 && j > LO && j < HI + 1)
      dev_fail(a.err, DERR_PRESSURE, task.slot, i, j, static_cast<double>(w[4]));
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 8; k++) bad |= bits_nan(w[k]);
    if (bad) dev_fail(a.err, DERR_NAN, task.slot, i, j, 0.0);
  }
}

// MUSCL2D.cpp:24-116 for one face of one leaf: x faces (i+1/2, j) for i, j in
// [LO, HI], then y faces (i, j+1/2).  On the FP64 path the kernels around it
// are bound by the FP64 pipe (76-80 % busy with 12 warps per SM): about 230
// FP64 instructions per MC + RUSA face and 330 per MC + HLLD face, all of them
// additions and multiplications (softfp.cuh takes the rest).
// False, with nothing stored or reported, if an operand left the range of the
// arithmetic M.
template <int NG, int RECON, int FLUX, typename S, class M>
__device__ __forceinline__ bool face_flux_with(const SplitArgs &a, size_t e) {
  using G = Geo<NG>;
  using T = S;
  constexpr int N = G::N, NN = G::NN, LO = G::LO, NF = G::NF, PER = 2 * NF * NF;
  const int t = static_cast<int>(e / PER), f = static_cast<int>(e % PER);
  const LeafTask task = a.tasks[t];
  const InstParams ip = a.inst[task.inst];
  const size_t base = static_cast<size_t>(task.slot) * 8 * NN;
  const S *W = static_cast<const S *>(a.W) + base;
  const bool yf = f >= NF * NF;
  const int g = yf ? f - NF * NF : f;
  const int r = g / NF, c = g % NF;
  const int s = yf ? N : 1;
  const int cL = (LO + r) * N + (LO + c);
  const T gamma = static_cast<T>(ip.gamma), h = static_cast<T>(yf ? task.dy : task.dx);
  const int fpos = cL + s;
  const double *Bf = a.B + static_cast<size_t>(task.slot) * 2 * NN + (yf ? NN : 0);
  const T bn = static_cast<T>(Bf[fpos]);
  S *out = static_cast<S *>(yf ? a.gg : a.ff) + base + fpos;
  T fl[8];
  M m;
  const int rc = face_flux_of<RECON, FLUX, NN, T>(m, W, cL, s, yf, ip.limiter, h, bn, gamma, fl);
  if (m.failed()) return false;
  if (rc) dev_fail(a.err, rc, task.slot, fpos % N, fpos / N, 0.0);
  bool bad = false;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    bad |= bits_nan(fl[k]);
    out[face_plane(k, yf) * NN] = fl[k];
  }
  if (bad) dev_fail(a.err, DERR_NAN, task.slot, fpos % N, fpos / N, 0.0);
  return true;
}

// the same with the native operators, for the rare face whose operands left
// the range of the Soft or Quick arithmetic; a function of its own, so that its
// registers are not the hot path's
template <int NG, int RECON, int FLUX, typename S>
__device__ __noinline__ void face_flux_native(const SplitArgs &a, size_t e) {
  face_flux_with<NG, RECON, FLUX, S, Native<S>>(a, e);
}
template <int NG, int RECON, int FLUX, typename S>
__device__ __forceinline__ void face_flux(const SplitArgs &a, size_t e) {
  if (!face_flux_with<NG, RECON, FLUX, S, typename FaceArith<S>::type>(a, e)) face_flux_native<NG, RECON, FLUX, S>(a, e);
}

template <int NG, int RECON, int FLUX, typename S, int MINB>
__global__ void __launch_bounds__(128, MINB) k_faces(const __grid_constant__ SplitArgs a) {
  pdl_wait();
  constexpr int PER = 2 * Geo<NG>::NF * Geo<NG>::NF;
  const size_t e = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= static_cast<size_t>(a.ntasks) * PER) return;
  face_flux<NG, RECON, FLUX, S>(a, e);
}

// persistent variant: a grid sized to the CTAs the SMs hold at once walks
// the whole face list of the step (all leaf blocks of all instances)
template <int NG, int RECON, int FLUX, typename S, int MINB>
__global__ void __launch_bounds__(128, MINB) k_faces_persist(const __grid_constant__ SplitArgs a) {
  pdl_wait();
  constexpr int PER = 2 * Geo<NG>::NF * Geo<NG>::NF;
  const size_t n = static_cast<size_t>(a.ntasks) * PER;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t e = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n; e += stride)
    face_flux<NG, RECON, FLUX, S>(a, e);
}

// persistent variant with dynamic work distribution: a grid of the CTAs the
// SMs hold at once, each warp claiming the next 32 faces of the step's face
// list from a global counter, so that a warp that was quick takes more; the
// last CTA to finish zeroes the counters for the next launch (every CTA has
// left its loop by then, so nothing claims work any more)
template <int NG, int RECON, int FLUX, typename S, int MINB>
__global__ void __launch_bounds__(128, MINB) k_faces_dyn(const __grid_constant__ SplitArgs a) {
  pdl_wait();
  constexpr int PER = 2 * Geo<NG>::NF * Geo<NG>::NF;
  const unsigned n = static_cast<unsigned>(a.ntasks) * PER;
  const int lane = threadIdx.x & 31;
  for (;;) {
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(&a.ctr[0], 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= n) break;
    if (base + lane < n) face_flux<NG, RECON, FLUX, S>(a, base + lane);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.ctr[1], 1u) == gridDim.x - 1) {
      a.ctr[0] = 0;
      a.ctr[1] = 0;
    }
  }
}

// Element r of a block's 8 x NN values in the order of k_resid: first the
// [LO, HI]^2 cells of the 8 variables, then the others (where the residual is
// zero), so that a warp is wholly one or the other.  Returns the index k*NN + c.
template <int NG>
__device__ __forceinline__ int resid_element(int r, bool &inside) {
  using G = Geo<NG>;
  constexpr int N = G::N, NN = G::NN, LO = G::LO, NF = G::NF, IN = NF * NF, OUT = NN - IN, SIDE = N - NF;
  inside = r < 8 * IN;
  if (inside) {
    const int k = r / IN, q = r % IN;
    return k * NN + (LO + q / NF) * N + LO + q % NF;
  }
  const int g = r - 8 * IN, k = g / OUT, q = g % OUT;
  if (q < LO * N) return k * NN + q;                        // rows below LO
  if (q < SIDE * N) return k * NN + q + NF * N;             // rows above HI
  const int m = q - SIDE * N, i = m % SIDE;                 // columns beside [LO, HI]
  return k * NN + (LO + m / SIDE) * N + (i < LO ? i : i + NF);
}

// residual on [LO, HI]^2 (zero elsewhere) and the RK stage on every cell
// (main.cpp:147-157 / 179-189).  Bound by the FP64 pipe (76-80 % busy): 5 FP64
// instructions per value in stage 1 and 6 in stage 2, the divisions by the
// cell size Soft (softfp.cuh) or, for power-of-two cells, on the exponent; a
// value outside [LO, HI]^2, whose residual is zero, takes none (1 in stage 2).
// The 256 blocks of an Orszag-Tang mesh with four ghost layers: 15 and 19 us
// (18 and 27 with every value on the same path; 59 and 71 with the compiler's
// divisions).
template <int NG, typename S>
__global__ void __launch_bounds__(512) k_resid(SplitArgs a) {
  pdl_wait();
  using G = Geo<NG>;
  using T = S;
  constexpr int N = G::N, NN = G::NN;
  const size_t e = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  // fused fill: the flux fill's snapshots (this kernel writes only qout)
  if (a.fuse.save.nseg) fill_save_all<N, S>(a.fuse, e, static_cast<size_t>(gridDim.x) * blockDim.x);
  if (e >= static_cast<size_t>(a.ntasks) * 8 * NN) return;
  const int t = static_cast<int>(e / (8 * NN));
  bool inside;
  const int r = resid_element<NG>(static_cast<int>(e % (8 * NN)), inside);
  const LeafTask &task = a.tasks[t];
  const size_t idx = static_cast<size_t>(task.slot) * 8 * NN + r;
  const T dt = static_cast<T>(a.inst[task.inst].dt);
  const T q = static_cast<const S *>(a.qin)[idx];
  S *out = static_cast<S *>(a.qout) + idx;
  const T old = a.step == 1 ? T(0) : *out;
  T d = T(0), v = T(0);   // dt * residual
  if (inside) {
    const S *ff = static_cast<const S *>(a.ff) + idx;
    const S *gg = static_cast<const S *>(a.gg) + idx;
    const T fx = ff[1] - ff[0], gy = gg[N] - gg[0];
    if (task.inv_dx != 0.0 && task.inv_dy != 0.0)  // power-of-two cells: exact reciprocal
      evaluate<T>([&](auto &m) {
        d = m.scaled(fx, static_cast<T>(task.inv_dx)) + m.scaled(gy, static_cast<T>(task.inv_dy));
      });
    else
      evaluate<T>([&](auto &m) { d = m.div(fx, static_cast<T>(task.dx)) + m.div(gy, static_cast<T>(task.dy)); });
    d = dt * d;
  }
  if (a.step == 1) v = inside ? q - d : q;
  else evaluate<T>([&](auto &m) { v = m.half(inside ? old + q - d : old + q); });
  *out = v;
}

}  // namespace amr
