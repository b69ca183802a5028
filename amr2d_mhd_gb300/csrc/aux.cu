// Launchers of the ghost-fill, CT, dt / criterion and refine / coarsen
// kernels, and the stage dispatcher.  Compiled without FMA contraction: the
// FP64 instantiations reproduce the reference's arithmetic.
#include "aux_kernels.cuh"
#include "launch.hpp"
#include "stage_split.cuh"

namespace amr {

bool method_supported(const Method &m) {
  if (m.flux < FLX_RUSA || m.flux > FLX_HLLD) return false;
  if (m.ng == 2) return m.recon == REC_MUSCL || m.recon == REC_WENO3;
  if (m.ng == 4) return m.recon == REC_MUSCL || m.recon == REC_WENO3 || m.recon == REC_WENO5;
  return false;
}

cudaError_t launch_stage(const Method &m, const StageArgs &a, int n, cudaStream_t s) {
  if (!method_supported(m)) return cudaErrorInvalidValue;
  if (!m.f32) {
    switch (m.flux) {
      case FLX_RUSA: return launch_stage_f64_rusa(m, a, n, s);
      case FLX_HLLE: return launch_stage_f64_hlle(m, a, n, s);
      case FLX_HLLC: return launch_stage_f64_hllc(m, a, n, s);
      default: return launch_stage_f64_hlld(m, a, n, s);
    }
  }
  switch (m.flux) {
    case FLX_RUSA: return launch_stage_f32_rusa(m, a, n, s);
    case FLX_HLLE: return launch_stage_f32_hlle(m, a, n, s);
    case FLX_HLLC: return launch_stage_f32_hllc(m, a, n, s);
    default: return launch_stage_f32_hlld(m, a, n, s);
  }
}

cudaError_t launch_faces(const Method &m, const SplitArgs &a, cudaStream_t s) {
  if (!method_supported(m)) return cudaErrorInvalidValue;
  if (!m.f32) {
    switch (m.flux) {
      case FLX_RUSA: return launch_faces_f64_rusa(m, a, s);
      case FLX_HLLE: return launch_faces_f64_hlle(m, a, s);
      case FLX_HLLC: return launch_faces_f64_hllc(m, a, s);
      default: return launch_faces_f64_hlld(m, a, s);
    }
  }
  switch (m.flux) {
    case FLX_RUSA: return launch_faces_f32_rusa(m, a, s);
    case FLX_HLLE: return launch_faces_f32_hlle(m, a, s);
    case FLX_HLLC: return launch_faces_f32_hllc(m, a, s);
    default: return launch_faces_f32_hlld(m, a, s);
  }
}

namespace {
int sm_count() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      sms = 0;
  }
  return sms;
}

// Up to two leaves per SM: the kernels with one CTA per leaf take 512 threads
// instead of 256, as their time is that of one leaf's rounds of cells (196
// leaves: k_prim_task 13.6 -> 12.6 us, FP32 k_dt_cell 10.3 -> 9.2; 40-leaf
// Brio-Wu program 6293 -> 6165 us with both)
bool wide_cta(int ntasks) { return ntasks <= 2 * sm_count(); }
int cell_threads(const Method &m) { return m.cell_block == 128 || m.cell_block == 512 ? m.cell_block : 256; }
}  // namespace

cudaError_t launch_prim(const Method &m, const SplitArgs &a, cudaStream_t s) {
  const int nn = m.ng == 2 ? Geo<2>::NN : Geo<4>::NN;
  const size_t n = static_cast<size_t>(a.ntasks) * nn;
  if (n == 0) return cudaSuccess;
  if (a.fuse.apply.nseg) {  // fused fill: one CTA per leaf
    const int w = wide_cta(a.ntasks) ? 512 : 256;
    if (m.ng == 2 && !m.f32) return launch_k(m.pdl, k_prim_task<2, double>, a.ntasks, w, 0, s, a);
    if (m.ng == 2) return launch_k(m.pdl, k_prim_task<2, float>, a.ntasks, w, 0, s, a);
    if (!m.f32) return launch_k(m.pdl, k_prim_task<4, double>, a.ntasks, w, 0, s, a);
    return launch_k(m.pdl, k_prim_task<4, float>, a.ntasks, w, 0, s, a);
  }
  const int b = cell_threads(m);
  const unsigned g = static_cast<unsigned>((n + b - 1) / b);
  if (m.ng == 2 && !m.f32) return launch_k(m.pdl, k_prim<2, double>, g, b, 0, s, a);
  if (m.ng == 2) return launch_k(m.pdl, k_prim<2, float>, g, b, 0, s, a);
  if (!m.f32) return launch_k(m.pdl, k_prim<4, double>, g, b, 0, s, a);
  return launch_k(m.pdl, k_prim<4, float>, g, b, 0, s, a);
}

cudaError_t launch_resid(const Method &m, const SplitArgs &a, cudaStream_t s) {
  const int nn = m.ng == 2 ? Geo<2>::NN : Geo<4>::NN;
  const size_t n = static_cast<size_t>(a.ntasks) * 8 * nn;
  if (n == 0) return cudaSuccess;
  const int b = cell_threads(m);
  const unsigned g = static_cast<unsigned>((n + b - 1) / b);
  if (m.ng == 2 && !m.f32) return launch_k(m.pdl, k_resid<2, double>, g, b, 0, s, a);
  if (m.ng == 2) return launch_k(m.pdl, k_resid<2, float>, g, b, 0, s, a);
  if (!m.f32) return launch_k(m.pdl, k_resid<4, double>, g, b, 0, s, a);
  return launch_k(m.pdl, k_resid<4, float>, g, b, 0, s, a);
}

cudaError_t launch_ghost(const Method &m, const GhostLaunch &in, cudaStream_t s) {
  const int B = m.ghost_block == 128 || m.ghost_block == 512 ? m.ghost_block : 256;
  const int ng = m.ng;
  GhostLaunch g = in;
  g.row0[0] = 0;
  for (int q = 0; q < g.nseg; q++) g.row0[q + 1] = g.row0[q] + g.seg[q].nv;
  const unsigned rows = static_cast<unsigned>(g.row0[g.nseg]);
  const dim3 gs((g.nsnaps + B - 1) / B, rows), go((g.nops + B - 1) / B, rows);
  if (g.nsnaps > 0 && rows > 0) {
    const cudaError_t e = ng == 2 ? launch_k(m.pdl, k_ghost_snap<Geo<2>::N>, gs, B, 0, s, g)
                                  : launch_k(m.pdl, k_ghost_snap<Geo<4>::N>, gs, B, 0, s, g);
    if (e != cudaSuccess) return e;
  }
  if (g.nops > 0 && rows > 0)
    return ng == 2 ? launch_k(m.pdl, k_ghost_apply<Geo<2>::N>, go, B, 0, s, g)
                   : launch_k(m.pdl, k_ghost_apply<Geo<4>::N>, go, B, 0, s, g);
  return cudaSuccess;
}

#define AMR_DISPATCH_NG_S(m, KERNEL, grid, block, smem, s, args)                 \
  do {                                                                            \
    if ((m).ng == 2 && !(m).f32) KERNEL<2, double><<<grid, block, smem, s>>>(args); \
    else if ((m).ng == 2) KERNEL<2, float><<<grid, block, smem, s>>>(args);       \
    else if (!(m).f32) KERNEL<4, double><<<grid, block, smem, s>>>(args);         \
    else KERNEL<4, float><<<grid, block, smem, s>>>(args);                        \
  } while (0)

// the same for the step's kernels, as programmatic dependents (Method::pdl)
#define AMR_DISPATCH_NG_S_PDL(m, KERNEL, grid, block, smem, s, args)                                          \
  (((m).ng == 2 && !(m).f32) ? launch_k((m).pdl, KERNEL<2, double>, dim3(grid), dim3(block), smem, s, args) \
   : ((m).ng == 2)           ? launch_k((m).pdl, KERNEL<2, float>, dim3(grid), dim3(block), smem, s, args)  \
   : !(m).f32                ? launch_k((m).pdl, KERNEL<4, double>, dim3(grid), dim3(block), smem, s, args) \
                             : launch_k((m).pdl, KERNEL<4, float>, dim3(grid), dim3(block), smem, s, args))

namespace {
// The widest CTAs with which all leaves are resident at once, else 128 threads:
// the 400 cells of a leaf take 1, 2 or 4 rounds.  KH meshes, us per step with
// the cooperative launch / 128 / 224 / 416 threads: FP32 16 leaves 79 / - / 76 /
// 72, 196: 90 / - / 86 / 82.5, 400: 134 / 111 / 100 / 95.5, 576: - / 121 / 113 /
// 124, 784: - / 146 / 142 / 149, 1024: 215 / 168 / 175 / 179, 4096: 754 / 574 / 589
// / 642; FP64 196: 236 / - / 232 / 230, 324: 352 / 343 / 334 / 340, 576: - / 541 /
// 532 / 539, 784: - / 725 / 729 / 732.
int ct_threads(const Method &m, int n) {
  for (const int t : {416, 224})
    if (n <= sm_count() * (m.f32 ? ct_resident<float>(t) : ct_resident<double>(t))) return t;
  return 128;
}
}  // namespace

#define AMR_CT_WIDTH(m, KERNEL, T, n, s, args)                                                             \
  (((m).ng == 2 && !(m).f32) ? launch_k((m).pdl, KERNEL<2, double, T>, dim3(n), dim3(T), 0, s, args)       \
   : ((m).ng == 2)           ? launch_k((m).pdl, KERNEL<2, float, T>, dim3(n), dim3(T), 0, s, args)        \
   : !(m).f32                ? launch_k((m).pdl, KERNEL<4, double, T>, dim3(n), dim3(T), 0, s, args)       \
                             : launch_k((m).pdl, KERNEL<4, float, T>, dim3(n), dim3(T), 0, s, args))
#define AMR_DISPATCH_CT(m, KERNEL, n, s, args)                                       \
  (ct_threads(m, n) == 416   ? AMR_CT_WIDTH(m, KERNEL, 416, n, s, args)              \
   : ct_threads(m, n) == 224 ? AMR_CT_WIDTH(m, KERNEL, 224, n, s, args)              \
                             : AMR_CT_WIDTH(m, KERNEL, 128, n, s, args))


cudaError_t launch_ct_emf(const Method &m, const CtArgs &a, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return AMR_DISPATCH_CT(m, k_ct_emf, n, s, a);
}

cudaError_t launch_ct_face(const Method &m, const CtArgs &a, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return AMR_DISPATCH_CT(m, k_ct_face, n, s, a);
}

// One cooperative launch (all CTAs resident: grid = SMs x resident CTAs per
// SM, capped at the task count), not a programmatic dependent.  512 threads
// per CTA: the phases of few leaves are rounds of dependent loads (rotor of 196
// leaves, us per pass with 128 / 256 / 512 threads: FP32 1500 / 1386 / 1281,
// FP64 1565 / 1515 / 1507).
cudaError_t launch_ct_coop(const Method &m, const CtArgs &a, const FillFuse &f_emf, const FillFuse &f_face,
                           const FillFuse &f_cell, unsigned *bar, cudaStream_t s) {
  if (a.ntasks <= 0) return cudaSuccess;
  static int per_sm[2][2] = {{0, 0}, {0, 0}};
  constexpr int threads = 512;
  void (*k)(CtArgs, FillFuse, FillFuse, FillFuse, unsigned *) =
      m.ng == 2 ? (m.f32 ? k_ct_coop<2, float, threads> : k_ct_coop<2, double, threads>)
                : (m.f32 ? k_ct_coop<4, float, threads> : k_ct_coop<4, double, threads>);
  int &ps = per_sm[m.ng == 2 ? 0 : 1][m.f32 ? 1 : 0];
  if (!ps) {
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps, k, threads, 0);
    if (e != cudaSuccess) return e;
    if (ps < 1) return cudaErrorInvalidConfiguration;
  }
  const int cap = sm_count() * ps;
  if (cap < 1) return cudaErrorInvalidDevice;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.ntasks < cap ? a.ntasks : cap);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, a, f_emf, f_face, f_cell, bar);
}

cudaError_t launch_diffuse(const Method &m, const CtArgs &a, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return AMR_DISPATCH_NG_S_PDL(m, k_diffuse, n, 128, 0, s, a);
}

cudaError_t launch_ct_cell(const Method &m, const CtArgs &a, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return AMR_DISPATCH_CT(m, k_ct_cell, n, s, a);
}

cudaError_t launch_dt_cell(const Method &m, const DtArgs &a, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (wide_cta(n)) return AMR_DISPATCH_NG_S_PDL(m, k_dt_cell_wide, n, 512, 0, s, a);
  return AMR_DISPATCH_NG_S_PDL(m, k_dt_cell, n, 256, 0, s, a);
}

cudaError_t launch_ic(const Method &m, const IcDev *blocks, int n, const double *tabs, void *U, double *Bi,
                      double *grad, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (m.ng == 2 && !m.f32) k_ic<2, double><<<n, 256, 0, s>>>(blocks, tabs, static_cast<double *>(U), Bi, grad);
  else if (m.ng == 2) k_ic<2, float><<<n, 256, 0, s>>>(blocks, tabs, static_cast<float *>(U), Bi, grad);
  else if (!m.f32) k_ic<4, double><<<n, 256, 0, s>>>(blocks, tabs, static_cast<double *>(U), Bi, grad);
  else k_ic<4, float><<<n, 256, 0, s>>>(blocks, tabs, static_cast<float *>(U), Bi, grad);
  return cudaGetLastError();
}

cudaError_t launch_refine(const Method &m, const TreeOpArgs &a, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int per = 4 * (m.ng == 2 ? refine_chunks<2>() : refine_chunks<4>());   // (son, chunk) CTAs per op
  AMR_DISPATCH_NG_S(m, k_refine, n * per, kRefineChunk, 0, s, a);
  return cudaGetLastError();
}

cudaError_t launch_coarsen(const Method &m, const TreeOpArgs &a, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  AMR_DISPATCH_NG_S(m, k_coarsen, n, 256, 0, s, a);
  return cudaGetLastError();
}

// Copy whole blocks between the slot pool and a dense float64 staging array
// (block b of the staging array <-> slot slots[b]), converting FP32 fields.
// blocks [0, nblk) of a field between the slot pool and a dense float64
// array [block][per] (device memory, or a host array the GPU addresses); two
// consecutive values per thread (`per` is even, so a pair never straddles
// blocks) when the dense array is 16-byte aligned
template <int W>
__global__ void k_gather(const int *slots, int nblk, const void *src, int f32, int per, double *dst) {
  const size_t total = static_cast<size_t>(nblk) * per / W;
  for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t i = e * W, b = i / per, r = i % per;
    const size_t s = static_cast<size_t>(slots[b]) * per + r;
    if (W == 2) {
      double2 v;
      if (f32) {
        const float2 f = *reinterpret_cast<const float2 *>(static_cast<const float *>(src) + s);
        v.x = f.x;
        v.y = f.y;
      } else {
        v = *reinterpret_cast<const double2 *>(static_cast<const double *>(src) + s);
      }
      *reinterpret_cast<double2 *>(dst + i) = v;
    } else {
      dst[i] = f32 ? static_cast<double>(static_cast<const float *>(src)[s]) : static_cast<const double *>(src)[s];
    }
  }
}

template <int W>
__global__ void k_scatter(const int *slots, int nblk, void *dst, int f32, int per, const double *src) {
  const size_t total = static_cast<size_t>(nblk) * per / W;
  for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t i = e * W, b = i / per, r = i % per;
    const size_t d = static_cast<size_t>(slots[b]) * per + r;
    if (W == 2) {
      const double2 v = *reinterpret_cast<const double2 *>(src + i);
      if (f32) *reinterpret_cast<float2 *>(static_cast<float *>(dst) + d) = make_float2(static_cast<float>(v.x),
                                                                                          static_cast<float>(v.y));
      else *reinterpret_cast<double2 *>(static_cast<double *>(dst) + d) = v;
    } else {
      if (f32) static_cast<float *>(dst)[d] = static_cast<float>(src[i]);
      else static_cast<double *>(dst)[d] = src[i];
    }
  }
}

namespace {
bool pairs_ok(const void *dense, int per) { return per % 2 == 0 && reinterpret_cast<uintptr_t>(dense) % 16 == 0; }
int xfer_grid(size_t items) { return static_cast<int>((items + 255) / 256 < 152 * 16 ? (items + 255) / 256 : 152 * 16); }
}  // namespace

cudaError_t launch_gather(const int *slots, int nblk, const void *src, int f32, int per, double *dst,
                          cudaStream_t s) {
  if (nblk <= 0) return cudaSuccess;
  const size_t total = static_cast<size_t>(nblk) * per;
  if (pairs_ok(dst, per)) k_gather<2><<<xfer_grid(total / 2), 256, 0, s>>>(slots, nblk, src, f32, per, dst);
  else k_gather<1><<<xfer_grid(total), 256, 0, s>>>(slots, nblk, src, f32, per, dst);
  return cudaGetLastError();
}

cudaError_t launch_scatter(const int *slots, int nblk, void *dst, int f32, int per, const double *src,
                           cudaStream_t s) {
  if (nblk <= 0) return cudaSuccess;
  const size_t total = static_cast<size_t>(nblk) * per;
  if (pairs_ok(src, per)) k_scatter<2><<<xfer_grid(total / 2), 256, 0, s>>>(slots, nblk, dst, f32, per, src);
  else k_scatter<1><<<xfer_grid(total), 256, 0, s>>>(slots, nblk, dst, f32, per, src);
  return cudaGetLastError();
}

}  // namespace amr
