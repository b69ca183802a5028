// Instantiates the stage or face kernels of one Riemann solver and one precision for
// every supported (ghost layers, reconstruction) pair.
#pragma once

#include "launch.hpp"
#include "stage.cuh"
#include "stage_split.cuh"

namespace amr {

// persistent = 2 (and a.ctr set): k_stage_dyn on a grid of the CTAs the SMs
// hold at once; otherwise one CTA per leaf block, the wide one for up to two FP32
// blocks per SM: with so few the launch lasts as long as one block, whose
// rounds of faces and cells it halves (196 blocks: 18 and 16 us against 26 and
// 24).
template <int NG, int RECON, int FLUX, typename S>
cudaError_t launch_stage_t(const StageArgs &a, int ntasks, int pdl, int persistent, cudaStream_t s) {
  constexpr int smem = stage_smem_bytes<NG, S>();
  constexpr int threads = StageShape<NG, S>::threads, wide = sizeof(S) == 4 ? kStageWide : threads;
  auto once = k_stage<NG, RECON, FLUX, S, threads>;
  auto once_wide = k_stage<NG, RECON, FLUX, S, wide>;
  auto dyn = k_stage_dyn<NG, RECON, FLUX, S>;
  static bool attr_set = false;
  static int per_sm = 0, sms = 0;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(once, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(once_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(dyn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int dev = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dyn, threads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    attr_set = true;
  }
  if (ntasks <= 0) return cudaSuccess;
  if (persistent == 2 && a.ctr) {
    const int grid = ntasks < sms * per_sm ? ntasks : sms * per_sm;
    return launch_k(pdl, dyn, grid, threads, smem, s, a);
  }
  if (wide != threads && ntasks <= 2 * sms) return launch_k(pdl, once_wide, ntasks, wide, smem, s, a);
  return launch_k(pdl, once, ntasks, threads, smem, s, a);
}

template <int FLUX, typename S>
cudaError_t launch_stage_flux(const Method &m, const StageArgs &a, int ntasks, cudaStream_t s) {
  const int p = m.persistent;
  if (m.ng == 2 && m.recon == REC_MUSCL) return launch_stage_t<2, REC_MUSCL, FLUX, S>(a, ntasks, m.pdl, p, s);
  if (m.ng == 2 && m.recon == REC_WENO3) return launch_stage_t<2, REC_WENO3, FLUX, S>(a, ntasks, m.pdl, p, s);
  if (m.ng == 4 && m.recon == REC_MUSCL) return launch_stage_t<4, REC_MUSCL, FLUX, S>(a, ntasks, m.pdl, p, s);
  if (m.ng == 4 && m.recon == REC_WENO3) return launch_stage_t<4, REC_WENO3, FLUX, S>(a, ntasks, m.pdl, p, s);
  if (m.ng == 4 && m.recon == REC_WENO5) return launch_stage_t<4, REC_WENO5, FLUX, S>(a, ntasks, m.pdl, p, s);
  return cudaErrorInvalidValue;
}

// Resident CTAs of 128 threads per SM the FP64-bound face kernels are compiled
// for: 4 (128 registers) for Rusanov and for WENO5, whose spills cost less
// than the fourth CTA brings (256^2 KH, MC + RUSA: 1547 against 1581 us per
// 4-step pass with 3; Orszag-Tang, WENO5 + HLLD: 1714 against 1821), 3 for
// the rest (rotor, MC + HLLD: 1610 against 1655 us with 4).  FP32: 8 (64
// registers; WENO5 6, 80), what the face itself takes; left free, the native
// repetition would set the kernel's registers, 68 to 127.
template <int RECON, int FLUX, typename S>
constexpr int faces_minb() {
  if (sizeof(S) == 4) return RECON == REC_WENO5 ? 6 : 8;
  return RECON == REC_WENO5 || FLUX == FLX_RUSA ? 4 : 3;
}

// persistent: 0 one CTA per `block` faces; 1 a grid of resident CTAs
// striding over the face list; 2 the same with dynamic claims of 32 faces
// per warp (k_faces_dyn, needs a.ctr)
template <int NG, int RECON, int FLUX, typename S>
cudaError_t launch_faces_t(const SplitArgs &a, int block, int persistent, int pdl, cudaStream_t s) {
  constexpr int PER = 2 * Geo<NG>::NF * Geo<NG>::NF;
  const size_t n = static_cast<size_t>(a.ntasks) * PER;
  if (n == 0) return cudaSuccess;
  // The one-shot kernel takes CTAs of one warp (its warps share nothing) unless
  // asked for 128 threads: they spread evenly and leave no SM waiting for a CTA's
  // last warp (rotor of 28 / 196 leaves, HLLD, 32.4 / 107 us against 34.4 / 109, 88
  // leaves of Brio-Wu, HLLE, 46.8 against 50.7, the same for Rusanov and WENO5).
  // The kernels are bounded at 128 threads per CTA.
  if (persistent) block = block == 64 ? 64 : 128;
  else block = block == 128 ? 128 : 32;
  size_t grid = (n + block - 1) / block;
  if (persistent == 2 && !a.ctr) persistent = 1;
  if (persistent) {
    // resident CTAs per SM for each (variant, block size), looked up once
    static int per_sm[2][2] = {{0, 0}, {0, 0}}, sms = 0;
    int &ps = per_sm[persistent == 2 ? 1 : 0][block == 64 ? 0 : 1];
    if (!sms) {
      int dev = 0;
      cudaError_t e = cudaGetDevice(&dev);
      if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess) return e;
    }
    if (!ps) {
      cudaError_t e = persistent == 2
          ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps, k_faces_dyn<NG, RECON, FLUX, S, (faces_minb<RECON, FLUX, S>())>,
                                                          block, 0)
          : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps, k_faces_persist<NG, RECON, FLUX, S, (faces_minb<RECON, FLUX, S>())>,
                                                          block, 0);
      if (e != cudaSuccess) return e;
      if (ps < 1) ps = 1;
    }
    const size_t cap = static_cast<size_t>(sms) * ps;
    if (grid > cap) grid = cap;
    if (persistent == 2)
      return launch_k(pdl, k_faces_dyn<NG, RECON, FLUX, S, (faces_minb<RECON, FLUX, S>())>, static_cast<unsigned>(grid), block, 0,
                      s, a);
    return launch_k(pdl, k_faces_persist<NG, RECON, FLUX, S, (faces_minb<RECON, FLUX, S>())>, static_cast<unsigned>(grid), block, 0,
                    s, a);
  }
  return launch_k(pdl, k_faces<NG, RECON, FLUX, S, (faces_minb<RECON, FLUX, S>())>, static_cast<unsigned>(grid), block, 0, s, a);
}

template <int FLUX, typename S>
cudaError_t launch_faces_flux(const Method &m, const SplitArgs &a, cudaStream_t s) {
  const int b = m.faces_block;
  const int p = m.persistent;
  if (m.ng == 2 && m.recon == REC_MUSCL) return launch_faces_t<2, REC_MUSCL, FLUX, S>(a, b, p, m.pdl, s);
  if (m.ng == 2 && m.recon == REC_WENO3) return launch_faces_t<2, REC_WENO3, FLUX, S>(a, b, p, m.pdl, s);
  if (m.ng == 4 && m.recon == REC_MUSCL) return launch_faces_t<4, REC_MUSCL, FLUX, S>(a, b, p, m.pdl, s);
  if (m.ng == 4 && m.recon == REC_WENO3) return launch_faces_t<4, REC_WENO3, FLUX, S>(a, b, p, m.pdl, s);
  if (m.ng == 4 && m.recon == REC_WENO5) return launch_faces_t<4, REC_WENO5, FLUX, S>(a, b, p, m.pdl, s);
  return cudaErrorInvalidValue;
}

}  // namespace amr

// the fused stage kernels and the face kernels of a solver and precision are
// translation units of their own (stage_*.cu, faces_*.cu), compiled in parallel
#define AMR_STAGE_DEFINE(P, F, FLUXID, T)                                                          \
  namespace amr {                                                                                  \
  cudaError_t launch_stage_##P##_##F(const Method &m, const StageArgs &a, int n, cudaStream_t s) { \
    return launch_stage_flux<FLUXID, T>(m, a, n, s);                                               \
  }                                                                                                \
  }
#define AMR_FACES_DEFINE(P, F, FLUXID, T)                                                   \
  namespace amr {                                                                           \
  cudaError_t launch_faces_##P##_##F(const Method &m, const SplitArgs &a, cudaStream_t s) { \
    return launch_faces_flux<FLUXID, T>(m, a, s);                                           \
  }                                                                                         \
  }
