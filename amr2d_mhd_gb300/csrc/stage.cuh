// Fused RK stage of one leaf block: MUSCL2D.cpp:13-121 (cons2prim,
// reconstruction, CT normal-B override, Riemann fluxes) followed by the
// residual and RK2ndv1 update of main.cpp:147-157 / 179-189.
//
// One CTA per leaf block.  Shared memory holds the primitive state of the
// whole block (with ghosts) and the x / y face fluxes that the residual
// needs; the fluxes also go to global memory (ff, gg), which the ghost fill
// and the CT EMF read next.
#pragma once

#include "amr_common.h"
#include "ghost.cuh"
#include "physics.cuh"

namespace amr {

template <int NG>
struct Geo {
  static constexpr int N = NI + 2 * NG;   // block edge with ghosts (nx of the reference)
  static constexpr int NN = N * N;
  static constexpr int LO = NG - 1;       // nxminb
  static constexpr int HI = NG + NI - 1;  // nxmax
  static constexpr int NF = NI + 1;       // faces per row computed by MUSCL2D (17)
  static constexpr int NFX = NI + 2;      // plus the stale face at LO (18)
};

struct StageArgs {
  const LeafTask *tasks;
  const InstParams *inst;
  const void *qin;    // U (stage 1) or Us (stage 2)
  void *qout;         // Us (stage 1) or U (stage 2, read-modify-write)
  const double *B;    // Bi (stage 1) or Bis (stage 2)
  void *ff;
  void *gg;
  DevError *err;
  unsigned *ctr;      // [2] block counter and finished-CTA counter of k_stage_dyn (zero between launches)
  int step;
  int ntasks;         // leaf blocks (k_stage_dyn)
  FillFuse fuse;      // fused fills: the qin fill gathered first (mirrored in
                      // shared memory), the flux fill's snapshots saved last
};

// First statement of every kernel of the step: when the kernel was launched
// as a programmatic dependent of the previous one (Method::pdl), wait until
// that grid has completed and its memory is visible; without that launch
// attribute it returns at once.  The kernel may then be scheduled while its
// predecessor drains, which hides most of the gap between the step's many
// small kernels.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The first failure is claimed in device memory and written to the record that
// the host reads after the step.  (A state that fails in every cell and face
// makes millions of claims: a step of 4096 blocks with 9.7 M of them takes 14 ms,
// 112 with the claims in host memory.)
__device__ __forceinline__ void dev_fail(DevError *e, int code, int blk, int i, int j, double v) {
  if (atomicCAS(&e->code, 0, code) == 0) {
    DevError *h = e->host;
    h->code = code;
    h->blk = blk;
    h->i = i;
    h->j = j;
    h->value = v;
  }
}

// floor of the pressure recovered by the FP32 path (code units)
constexpr float kPressureFloor = 1.0e-10f;

// gamma as the primitive recovery of storage type S takes it
template <typename S> struct GasGamma;
template <> struct GasGamma<double> {
  double g;
  __device__ __forceinline__ GasGamma(const InstParams &p) : g(p.gamma) {}
  __device__ __forceinline__ explicit GasGamma(double gamma) : g(gamma) {}
};
template <> struct GasGamma<float> {
  float hi, lo;   // gamma - 1
  __device__ __forceinline__ GasGamma(const InstParams &p) : hi(p.gm1_hi), lo(p.gm1_lo) {}
};

// meshblock.cpp:119-179 for one cell; the FP32 path recovers the pressure
// from pairs of floats and floors it (positivity fix).
template <typename S>
__device__ __forceinline__ void cons2prim_cell(const S *u, S *w, const GasGamma<S> &gam);

template <class M>
__device__ __forceinline__ void cons2prim_f64(M &m, const double *u, double *w, double g) {
  w[0] = u[0];
  w[1] = m.div(u[1], u[0]);
  w[2] = m.div(u[2], u[0]);
  w[3] = m.div(u[3], u[0]);
  double p = (g - 1) * (u[4] - m.half(w[0]) * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]));
  w[5] = u[5];
  w[6] = u[6];
  w[7] = u[7];
  w[4] = p - (g - 1) * m.half(u[5] * u[5] + u[6] * u[6] + u[7] * u[7]);
}
template <>
__device__ __forceinline__ void cons2prim_cell<double>(const double *u, double *w, const GasGamma<double> &gam) {
  evaluate<double>([&](auto &m) { cons2prim_f64(m, u, w, gam.g); });
}

// Pairs of floats.  The _rn intrinsics keep the compiler from fusing or
// reordering the steps.
// a + b = s + e exactly (Knuth's TwoSum)
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  const float v = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v));
}
// a^2 + b^2 + c^2 as hi + lo, exact to about 2^-48 relative: each square split
// exactly by an FMA (Dekker's product), the partial sums by TwoSum, with the
// error terms summed in FP32
__device__ __forceinline__ void sum_sq3(float a, float b, float c, float &hi, float &lo) {
  const float pa = __fmul_rn(a, a), pb = __fmul_rn(b, b), pc = __fmul_rn(c, c);
  const float ea = __fmaf_rn(a, a, -pa), eb = __fmaf_rn(b, b, -pb), ec = __fmaf_rn(c, c, -pc);
  float s1, t1, t2;
  two_sum(pa, pb, s1, t1);
  two_sum(s1, pc, hi, t2);
  lo = __fadd_rn(__fadd_rn(__fadd_rn(ea, eb), ec), __fadd_rn(t1, t2));
}

// FP32 path: the pressure from the total energy, (gamma - 1) (E - (|m|^2/rho +
// |B|^2)/2), whose cancellation is where FP32 loses digits, evaluated with
// unevaluated sums of floats: the sums of squares (sum_sq3) and |m|^2/rho with
// 1/rho = ir + rl (rl from the FMA residual 1 - rho*ir) as pairs, good to 2^-47 of
// their value; their sum and the subtraction without further error (TwoSum, also
// of the low parts, whose rounding would add half as much again); and the
// product with gamma - 1 (a pair as well).  The error is that of the same pairs
// summed in FP64 (rms 0.17-0.39 2^-48 of the subtracted terms, results within
// 0.5 ulp where they do not cancel), but no instruction is on the FP64 pipe,
// 12 of which per cell kept the FP32 path's dt kernel 76 % bound (16 clocks per
// warp each).  The velocities are the FP32 momenta times the FP32 reciprocal.
// (A component above ~1.8e19 overflows its FP32 square; such a state is out of
// the FP32 path's range in any case.)
template <>
__device__ __forceinline__ void cons2prim_cell<float>(const float *u, float *w, const GasGamma<float> &gam) {
  const float ir = 1.0f / u[0];
  const float rl = __fmul_rn(__fmaf_rn(-u[0], ir, 1.0f), ir);
  float mh, ml, bh, bl;
  sum_sq3(u[1], u[2], u[3], mh, ml);
  sum_sq3(u[5], u[6], u[7], bh, bl);
  const float kh = __fmul_rn(mh, ir);
  const float kl = __fadd_rn(__fmaf_rn(mh, ir, -kh), __fadd_rn(__fmul_rn(mh, rl), __fmul_rn(ml, ir)));
  // |m|^2/rho + |B|^2 = sh + s2 + e1 + e2, E - half of it = th + tl
  float sh, sl, s1, e1, s2, e2, dh, dl, th, tl;
  two_sum(kh, bh, sh, sl);
  two_sum(kl, bl, s1, e1);
  two_sum(sl, s1, s2, e2);
  two_sum(u[4], __fmul_rn(-0.5f, sh), dh, dl);
  two_sum(dh, __fmaf_rn(-0.5f, s2, dl), th, tl);
  tl = __fmaf_rn(-0.5f, __fadd_rn(e1, e2), tl);
  const float ph = __fmul_rn(gam.hi, th);
  float p = __fadd_rn(ph, __fadd_rn(__fmaf_rn(gam.hi, th, -ph), __fmaf_rn(gam.hi, tl, __fmul_rn(gam.lo, th))));
  // positivity fix of the FP32 path: the FP32 conserved state can put the
  // recovered pressure below zero where the FP64 path stays positive
  if (!(p > kPressureFloor)) p = kPressureFloor;
  w[0] = u[0];
  w[1] = u[1] * ir;
  w[2] = u[2] * ir;
  w[3] = u[3] * ir;
  w[4] = p;
  w[5] = u[5];
  w[6] = u[6];
  w[7] = u[7];
}

// ------------------------------------------------------------ bulk staging
// One thread issues a bulk copy (TMA, cp.async.bulk) of `bytes` contiguous
// bytes from global to shared memory, completing on an mbarrier; every
// thread then waits for the phase with a bounded spin.  Both addresses and
// the size are multiples of 16 bytes (checked by the caller's layout).
constexpr long kBulkSpinLimit = 1L << 26;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void bulk_stage_issue(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  const uint32_t b = smem_u32(bar);
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(b)
               : "memory");
}

// true once the phase completed; false after the spin limit
__device__ __forceinline__ bool bulk_stage_wait(uint64_t *bar, uint32_t phase) {
  const uint32_t b = smem_u32(bar);
  for (long it = 0; it < kBulkSpinLimit; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(b), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

// plane of variable k of the face frame (normal, tangential, z): riemannS
// rotates a y face (riemannS.cpp:12-23, 47-55), u <-> v and Bx <-> By
__device__ __forceinline__ int face_plane(int k, bool yf) {
  const int r = k == 1 ? 2 : k == 2 ? 1 : k == 5 ? 6 : k == 6 ? 5 : k;
  return yf ? r : k;
}

// The left and right MUSCL states of a face, variables 0-4, 6, 7 of the face
// frame, with one limiter
template <int LIM, int NN, typename T, class M>
__device__ __forceinline__ void muscl_states_of(M &m, const T *W, int cL, int s, bool yf, T h, T *wl, T *wr) {
#pragma unroll
  for (int k = 0; k < 8; k++) {
    if (k == 5) continue;
    const T *w = W + face_plane(k, yf) * NN + cL;
    const T wm = w[-s], w0 = w[0], w1 = w[s], w2 = w[2 * s];
    muscl_face<T>(m, LIM, w0, w1, w0 - wm, w1 - w0, w2 - w1, h, wl[k], wr[k]);
  }
}
// The limiter is picked once per face, outside the loop over the variables: a
// switch in the loop puts the variables' divisions one after the other (KH
// layer of 32 x 32 roots, HLLD, us per step: FP32 minmod 197 -> 185, Koren 199 ->
// 188; FP64 minmod 1125 -> 1087, Koren 1318 -> 1216).
template <int NN, typename T, class M>
__device__ __forceinline__ void muscl_states(M &m, const T *W, int cL, int s, bool yf, int lim, T h, T *wl, T *wr) {
  switch (lim) {
    case LIM_NOSL: muscl_states_of<LIM_NOSL, NN, T>(m, W, cL, s, yf, h, wl, wr); break;
    case LIM_MINMOD: muscl_states_of<LIM_MINMOD, NN, T>(m, W, cL, s, yf, h, wl, wr); break;
    case LIM_VANLEER: muscl_states_of<LIM_VANLEER, NN, T>(m, W, cL, s, yf, h, wl, wr); break;
    case LIM_SUPERBEE: muscl_states_of<LIM_SUPERBEE, NN, T>(m, W, cL, s, yf, h, wl, wr); break;
    case LIM_MC: muscl_states_of<LIM_MC, NN, T>(m, W, cL, s, yf, h, wl, wr); break;
    case LIM_KOREN: muscl_states_of<LIM_KOREN, NN, T>(m, W, cL, s, yf, h, wl, wr); break;
    case LIM_CADA3RD: muscl_states_of<LIM_CADA3RD, NN, T>(m, W, cL, s, yf, h, wl, wr); break;
    default: muscl_states_of<LIM_1ST, NN, T>(m, W, cL, s, yf, h, wl, wr); break;
  }
}

// MUSCL2D.cpp:24-116 for one face: W is plane 0 of the block's primitive
// state (planes NN apart), cL the cell on its left (below it), s the cell
// stride along its normal, yf whether that is y; bn the face's own normal
// field (the CT override, MUSCL2D.cpp:48-51).  The states are read and the
// flux is returned in the face frame, so that x and y faces of a warp run
// the same code.  Returns riemann()'s code.
template <int RECON, int FLUX, int NN, typename T, class M>
__device__ __forceinline__ int face_flux_of(M &m, const T *W, int cL, int s, bool yf, int lim, T h, T bn, T gamma,
                                            T *fl) {
  T wl[8], wr[8];
  if (RECON == REC_MUSCL) muscl_states<NN, T>(m, W, cL, s, yf, lim, h, wl, wr);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    if (RECON == REC_MUSCL || k == 5) continue;
    const T *w = W + face_plane(k, yf) * NN + cL;
    if (RECON == REC_WENO3) {
      T dummy;
      weno3_cell<T>(m, w[-s], w[0], w[s], wl[k], dummy);
      weno3_cell<T>(m, w[0], w[s], w[2 * s], dummy, wr[k]);
    } else {
      wl[k] = weno5_cell<T, false>(m, w[-2 * s], w[-s], w[0], w[s], w[2 * s]);
      wr[k] = weno5_cell<T, true>(m, w[-s], w[0], w[s], w[2 * s], w[3 * s]);
    }
  }
  wl[5] = bn;
  wr[5] = bn;
  return riemann<FLUX, T>(m, wl, wr, gamma, fl);
}

// Threads of the fused stage's CTA and resident CTAs per SM it is compiled for.
// FP32: 256 and 5 (48 registers), with four ghost layers 320 and 4.  The kernel
// issues in half of its cycles and waits on latency between its phases, so
// residents pay, up to the registers.  One GB300, us per pass of 32 rotors (12
// steps), 24 blasts (10 steps) and a 512^2 KH layer (8 steps), state transfers
// included:
//   256 threads x 5 CTAs  16342  6598  1768      320 x 4  16737  6730  1794
//   192 x 6               16448  6713  1831      320 x 3  17460  6966  1855
// and per step of a WENO5 + HLLD layer of 18 x 18 / 21 x 21 / 25 x 25 / 40 x 40
// blocks: 256 x 5 112 / 117 / 154 / 340, 320 x 4 108 / 113 / 157 / 336.
template <int NG, typename S> struct StageShape { static constexpr int threads = 256, min_blocks = 1; };
template <> struct StageShape<2, float> { static constexpr int threads = 256, min_blocks = 5; };
template <> struct StageShape<4, float> { static constexpr int threads = 320, min_blocks = 4; };

// variable 0 of face f of the block in shared memory
template <int NG, typename S>
__device__ __forceinline__ S *face_slot(S *sFx, S *sFy, int f) {
  constexpr int NF = Geo<NG>::NF, NFX = Geo<NG>::NFX;
  const int g = f >= NF * NF ? f - NF * NF : f, r = g / NF, c = g % NF;
  return f >= NF * NF ? sFy + (r + 1) * NF + c : sFx + r * NFX + c + 1;
}

// One face of the fused stage, evaluated with the arithmetic M: its flux to the
// block's faces in shared memory and to ff / gg.  False, with nothing stored
// or reported, if an operand left M's range.
template <int NG, int RECON, int FLUX, typename S, class M>
__device__ __forceinline__ bool stage_face(const StageArgs &a, const LeafTask &task, const S *sW, S *sFx, S *sFy,
                                           int lim, S gamma, int f) {
  using G = Geo<NG>;
  constexpr int N = G::N, NN = G::NN, LO = G::LO, NF = G::NF, NFX = G::NFX;
  const bool yf = f >= NF * NF;
  const int g = yf ? f - NF * NF : f;
  const int r = g / NF, c = g % NF;
  // cell-index stride along the face normal and the left cell of the face
  const int s = yf ? N : 1;
  const int cL = (LO + r) * N + (LO + c);
  const int fpos = cL + s;  // face index of the reference = the right cell
  const S h = static_cast<S>(yf ? task.dy : task.dx);
  const S bn = static_cast<S>(a.B[static_cast<size_t>(task.slot) * 2 * NN + (yf ? NN : 0) + fpos]);
  S fl[8];
  M m;
  const int rc = face_flux_of<RECON, FLUX, NN, S>(m, sW, cL, s, yf, lim, h, bn, gamma, fl);
  if (m.failed()) return false;
  if (rc) dev_fail(a.err, rc, task.slot, fpos % N, fpos / N, 0.0);
  S *out = static_cast<S *>(yf ? a.gg : a.ff) + static_cast<size_t>(task.slot) * 8 * NN + fpos;
  bool bad = false;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    bad |= bits_nan(fl[k]);
    const int p = face_plane(k, yf);
    if (!yf) sFx[(p * NF + r) * NFX + (c + 1)] = fl[k];
    else sFy[(p * NFX + (r + 1)) * NF + c] = fl[k];
    out[p * NN] = fl[k];
  }
  if (bad) dev_fail(a.err, DERR_NAN, task.slot, fpos % N, fpos / N, 0.0);
  return true;
}
// the same with the native operators, for the rare face whose operands left
// the range of the Soft or Quick arithmetic, with its arguments read again.
// FP64 calls it as a function of its own from the loop over the faces; FP32 has
// it inline after the loop, as the registers kept for a call cost batches 1 %.
template <int NG, int RECON, int FLUX, typename S>
__device__ __forceinline__ void stage_face_native(const StageArgs &a, int ti, const S *sW, S *sFx, S *sFy, int f) {
  const LeafTask task = a.tasks[ti];
  const InstParams ip = a.inst[task.inst];
  stage_face<NG, RECON, FLUX, S, Native<S>>(a, task, sW, sFx, sFy, ip.limiter, static_cast<S>(ip.gamma), f);
}
template <int NG, int RECON, int FLUX, typename S>
__device__ __noinline__ void stage_face_call(const StageArgs &a, int ti, const S *sW, S *sFx, S *sFy, int f) {
  stage_face_native<NG, RECON, FLUX, S>(a, ti, sW, sFx, sFy, f);
}

// One leaf block of the fused stage: task `ti`, its conserved state staged
// into shared memory by a bulk copy completing on `bar` (initialised by the
// caller) in phase `phase`.  Returns false (after recording DERR_TIMEOUT and
// letting the copy land) when the bounded wait gave up; the decision is the
// same in every thread of the CTA.
template <int NG, int RECON, int FLUX, typename S, bool PRE>
__device__ __forceinline__ bool stage_block(const StageArgs &a, int ti, uint64_t *bar, uint32_t phase) {
  using G = Geo<NG>;
  using T = S;
  constexpr int N = G::N, NN = G::NN, LO = G::LO, HI = G::HI, NF = G::NF, NFX = G::NFX;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *sW = reinterpret_cast<T *>(smem_raw);   // [8][NN]
  T *sFx = sW + 8 * NN;                      // [8][NF][NFX]   face i = LO + col, row j = LO + r
  T *sFy = sFx + 8 * NF * NFX;               // [8][NFX][NF]   face j = LO + row, col i = LO + c
  S *sU = sW;   // [8][NN] the conserved state, staged where the primitive state replaces it

  const LeafTask task = a.tasks[ti];
  const InstParams ip = a.inst[task.inst];
  const size_t base = static_cast<size_t>(task.slot) * 8 * NN;
  const S *Q = static_cast<const S *>(a.qin) + base;
  S *ff = static_cast<S *>(a.ff) + base;
  S *gg = static_cast<S *>(a.gg) + base;
  const double *Bx = a.B + static_cast<size_t>(task.slot) * 2 * NN;
  const double *By = Bx + NN;
  const int tid = block_tid(), nthr = blockDim.x;

  // 0. the block's conserved state (8 planes, contiguous) into shared memory by TMA
  static_assert((8 * NN * sizeof(S)) % 16 == 0, "bulk copies move multiples of 16 bytes");
  if (tid == 0) bulk_stage_issue(sU, Q, static_cast<uint32_t>(8 * NN * sizeof(S)), bar);
  // fused fill: each thread's first gathers are loaded while the copy is in
  // flight (not in the loop of k_stage_dyn, where the values held over the wait
  // spill)
  FillPre<S> pre;
  pre.on = false;
  if (PRE) fill_prefetch<N, S>(a.fuse, task, tid, pre);
  const bool late = !bulk_stage_wait(bar, phase);
  if (__syncthreads_or(late)) {
    if (tid == 0) dev_fail(a.err, DERR_TIMEOUT, task.slot, 0, 0, 0.0);
    bulk_stage_wait(bar, phase);  // let the copy land before the CTA's shared memory is released
    return false;
  }
  // fused fill: the block's ghost cells of qin (and of B), into global memory
  // and over the staged copy, which held the values from before the fill
  if (a.fuse.apply.nseg) {
    fill_apply_task_after<N, S>(a.fuse, task, tid, nthr, sU, pre);
    __syncthreads();
  }

  // 1. primitive variables of every cell (U2W / Us2W), with the traps (in
  // place unless the conserved state is kept)
  for (int c = tid; c < NN; c += nthr) {
    S u[8], w[8];
#pragma unroll
    for (int k = 0; k < 8; k++) u[k] = sU[k * NN + c];
    cons2prim_cell<S>(u, w, GasGamma<S>(ip));
#pragma unroll
    for (int k = 0; k < 8; k++) sW[k * NN + c] = w[k];
    const int i = c % N, j = c / N;
    if (w[4] <= T(0) && i > LO && i < HI + 1 && j > LO && j < HI + 1)
      dev_fail(a.err, DERR_PRESSURE, task.slot, i, j, static_cast<double>(w[4]));
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 8; k++) bad |= bits_nan(w[k]);
    if (bad) dev_fail(a.err, DERR_NAN, task.slot, i, j, 0.0);
  }
  // fluxes MUSCL2D does not recompute: the x face at LO and the y face at LO
  // (their values come from the previous ghost fill of ff / gg)
  for (int e = tid; e < 8 * NF; e += nthr) {
    const int k = e / NF, r = e % NF;
    sFx[(k * NF + r) * NFX + 0] = ff[k * NN + (LO + r) * N + LO];
    sFy[(k * NFX + 0) * NF + r] = gg[k * NN + LO * N + (LO + r)];
  }
  __syncthreads();

  // 2. Riemann fluxes at x faces (i+1/2, j), i in [LO, HI], and y faces
  const T gamma = static_cast<T>(ip.gamma);
  const int lim = ip.limiter;
  // FP32 faces to be repeated are marked by a NaN and taken after the loop
  bool again = false;
  for (int f = tid; f < 2 * NF * NF; f += nthr)
    if (!stage_face<NG, RECON, FLUX, S, typename FaceArith<S>::type>(a, task, sW, sFx, sFy, lim, gamma, f)) {
      if (sizeof(S) == 8) {
        stage_face_call<NG, RECON, FLUX, S>(a, ti, sW, sFx, sFy, f);
      } else {
        again = true;
        *face_slot<NG>(sFx, sFy, f) = T(NAN);
      }
    }
  if (sizeof(S) == 8) {
    __syncthreads();
  } else if (__syncthreads_or(again)) {
    for (int f = tid; f < 2 * NF * NF; f += nthr)
      if (bits_nan(*face_slot<NG>(sFx, sFy, f))) stage_face_native<NG, RECON, FLUX, S>(a, ti, sW, sFx, sFy, f);
    __syncthreads();
  }

  // 3. residual on [LO, HI]^2 (zero elsewhere) and the RK stage on every cell
  const T dt = static_cast<T>(ip.dt);
  // FP32: the rounded reciprocals once per block (a division per value has
  // no less error); FP64: the reference's divisions
  const T dx = static_cast<T>(sizeof(T) == 4 ? task.rcp_dx : task.dx);
  const T dy = static_cast<T>(sizeof(T) == 4 ? task.rcp_dy : task.dy);
  S *out = static_cast<S *>(a.qout) + base;
  for (int c = tid; c < NN; c += nthr) {   // all variables of a cell per thread: its index is decoded once
    const int i = c % N, j = c / N;
    const bool inside = i >= LO && i <= HI && j >= LO && j <= HI;
    const T *fx = sFx + (inside ? (j - LO) * NFX + i - LO : 0), *fy = sFy + (inside ? (j - LO) * NF + i - LO : 0);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      T res = T(0.);
      if (inside) {
        const T gx = fx[k * NF * NFX + 1] - fx[k * NF * NFX], gy = fy[k * NFX * NF + NF] - fy[k * NFX * NF];
        if (sizeof(T) == 4) res = gx * dx + gy * dy;
        else evaluate<T>([&](auto &m) { res = m.div(gx, dx) + m.div(gy, dy); });
      }
      const int e = k * NN + c;
      const T q = Q[e];
      if (a.step == 1) out[e] = q - dt * res;                         // Us = U - dt res
      else out[e] = T(0.5) * (out[e] + q - dt * res);                 // U = (U + Us - dt res)/2
    }
  }
  // fused fill: snapshots of the next fill (ff, gg and B, whose writes by
  // this CTA precede the barrier after step 2)
  if (a.fuse.save.nseg) fill_save_task<N, S>(a.fuse, task, tid, nthr);
  return true;
}

__device__ __forceinline__ void stage_bar_init(uint64_t *bar) {
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}

// One CTA per leaf block.  THREADS: StageShape's, or kStageWide for FP32 and
// few blocks, whose 640 threads take the 578 faces in one round.
constexpr int kStageWide = 640;
template <int NG, int RECON, int FLUX, typename S, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == kStageWide ? 2 : StageShape<NG, S>::min_blocks) k_stage(const __grid_constant__ StageArgs a) {
  pdl_wait();
  __shared__ __align__(8) uint64_t bar;
  stage_bar_init(&bar);
  stage_block<NG, RECON, FLUX, S, true>(a, blockIdx.x, &bar, 0);
}

// persistent: a grid of the CTAs the SMs hold at once sweeps the leaf list of
// all instances and levels, each CTA claiming the next block from a global
// counter (the mbarrier phase alternates per block); the last CTA to finish
// zeroes the counters for the next launch
template <int NG, int RECON, int FLUX, typename S>
__global__ void __launch_bounds__(StageShape<NG, S>::threads, StageShape<NG, S>::min_blocks) k_stage_dyn(const __grid_constant__ StageArgs a) {
  pdl_wait();
  __shared__ __align__(8) uint64_t bar;
  __shared__ int next;
  stage_bar_init(&bar);
  for (uint32_t it = 0;; it++) {
    if (threadIdx.x == 0) next = static_cast<int>(atomicAdd(&a.ctr[0], 1u));
    __syncthreads();
    const int ti = next;
    if (ti >= a.ntasks) break;
    if (!stage_block<NG, RECON, FLUX, S, false>(a, ti, &bar, it & 1u)) break;
    __syncthreads();  // shared memory free for the next block's copy
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.ctr[1], 1u) == gridDim.x - 1) {
      a.ctr[0] = 0;
      a.ctr[1] = 0;
    }
  }
}

template <int NG, typename S>
constexpr int stage_smem_bytes() {
  using G = Geo<NG>;
  return static_cast<int>(sizeof(S)) * (8 * G::NN + 2 * 8 * G::NF * G::NFX);
}

}  // namespace amr
