// Device side of the compiled ghost fills (ghost_compile.cpp): the gather of
// one op, the stand-alone fill launch, and the fused form in which a fill's
// gathers run in the kernel that consumes the filled field and its
// snapshots in the kernel before it.
#pragma once

#include <stddef.h>

#include <type_traits>

#include "amr_common.h"

namespace amr {

// One compiled program (ops + snapshots) serves every field; a launch applies
// it to up to kMaxSeg fields at once.
constexpr int kMaxSeg = 3;
struct GhostSeg {
  void *field;
  int nv;
  int kind;           // FILL_CC / FILL_FC / FILL_EC (ghost_compile.hpp)
  int f32;            // field stored as float
};
struct GhostLaunch {
  const GhostOp *ops;
  const GhostSnap *snaps;
  int nops, nsnaps;
  GhostSeg seg[kMaxSeg];
  int nseg;
  double *snapbuf;    // [nseg][nsnaps][8], values of the segment's type (snap_rows)
  // variable rows of the launch: segment q owns rows [row0[q], row0[q+1]);
  // set by launch_ghost
  int row0[kMaxSeg + 1];
  // the snapshots that begin a step also take its parameters from pinned host
  // memory to the device (nparams 0: not)
  const InstParams *params_from;
  InstParams *params_to;
  int nparams;
};

// A fill kernel runs on a 2-D grid: blockIdx.y is the variable row, so that
// consecutive threads take consecutive items (ops or snapshots) of the same
// variable and every load of an item is independent of the others.  The
// segment is picked with constant indices into the parameter block.
__device__ __forceinline__ GhostSeg ghost_seg(const GhostLaunch &g, int row, int &q, int &k) {
  GhostSeg s = g.seg[0];
  q = 0;
  k = row;
  if (g.nseg > 1 && row >= g.row0[1]) { s = g.seg[1]; q = 1; k = row - g.row0[1]; }
  if (g.nseg > 2 && row >= g.row0[2]) { s = g.seg[2]; q = 2; k = row - g.row0[2]; }
  return s;
}

// fine-to-coarse value of one variable from the patch (i,j) (i,j+1) (i+1,j)
// (i+1,j+1): boundary.cpp:48 / boundaryfc.cpp:48 / boundaryec.cpp:46
template <typename F>
__device__ __forceinline__ F fine_value(int kind, int k, F a00, F a01, F a10, F a11) {
  F v = F(0.);
  if (kind == 0) {
    v += a00; v += a01; v += a10; v += a11;
    return F(0.25) * v;
  }
  if (kind == 1) {
    v += a00;
    v += k == 0 ? a01 : a10;
    return F(0.5) * v;
  }
  return a00;
}

// the value(s) of variable k of one gather, computed in the field's type F
// (a pair gives two); and their store to the destination and, when `tile` is
// not null, to the destination block's copy of the field in shared memory
// ([nv][N*N])
template <int N, typename F>
__device__ __forceinline__ void ghost_gather(const GhostSeg &s, const GhostOp &op, int k, const F *snap, F &v0,
                                             F &v1) {
  constexpr int NN = N * N;
  const F *fld = static_cast<const F *>(s.field);
  if (op.type == GOP_COPY2) {  // even positions in an even-sized plane: aligned pair
    using P2 = typename std::conditional<sizeof(F) == 4, float2, double2>::type;
    const P2 v =
        *reinterpret_cast<const P2 *>(fld + (static_cast<size_t>(op.src_slot) * s.nv + k) * NN + op.src_pos);
    v0 = v.x;
    v1 = v.y;
    return;
  }
  if (op.type == GOP_COPY || op.type == GOP_FINE) {
    const F *c = fld + (static_cast<size_t>(op.src_slot) * s.nv + k) * NN + op.src_pos;
    v0 = op.type == GOP_COPY ? c[0] : fine_value<F>(s.kind, k, c[0], c[N], c[1], c[1 + N]);
  } else {
    const F *r = snap + static_cast<size_t>(op.src_slot) * 8 + k;
    v0 = op.type == GOP_SNAP ? r[0] : fine_value<F>(s.kind, k, r[0], r[8], r[16], r[24]);
  }
}

template <int N, typename F>
__device__ __forceinline__ void ghost_put(const GhostSeg &s, const GhostOp &op, int k, F v0, F v1, F *tile) {
  constexpr int NN = N * N;
  F *dst = static_cast<F *>(s.field) + (static_cast<size_t>(op.dst_slot) * s.nv + k) * NN + op.dst_pos;
  if (op.type == GOP_COPY2) {
    using P2 = typename std::conditional<sizeof(F) == 4, float2, double2>::type;
    P2 v;
    v.x = v0;
    v.y = v1;
    *reinterpret_cast<P2 *>(dst) = v;
    if (tile) *reinterpret_cast<P2 *>(tile + k * NN + op.dst_pos) = v;
    return;
  }
  *dst = v0;
  if (tile) tile[k * NN + op.dst_pos] = v0;
}

// A snapshot row holds 8 values of the field's own type (no conversion of
// FP32 values to double and back on the FP64 pipe); segment q's rows start at
// q * nsnaps rows of 8 doubles.
template <typename F>
__device__ __forceinline__ F *snap_rows(double *snapbuf, int q, int nsnaps) {
  return reinterpret_cast<F *>(snapbuf + static_cast<size_t>(q) * nsnaps * 8);
}

// variable k of one gather (`tile` as for ghost_put)
template <int N, typename F>
__device__ __forceinline__ void ghost_apply_one(const GhostSeg &s, const GhostOp &op, int k, const F *snap,
                                                F *tile = nullptr) {
  F v0, v1 = F(0.);
  ghost_gather<N, F>(s, op, k, snap, v0, v1);
  ghost_put<N, F>(s, op, k, v0, v1, tile);
}

// ------------------------------------------------------------ fused fills
// The compiled program is grouped by block: the ops that write block b's
// ghost cells are ops[op_begin, op_begin + op_count) of b's LeafTask, and
// the snapshots of b's cells snaps[snap_begin, snap_begin + snap_count).
// No op reads a cell that the same fill writes (those reads go through the
// snapshots), and every kernel of the step writes only the cells of its own
// block.  So a fill can run inside the kernel that consumes the field, each
// CTA gathering its own block's ghost cells first, provided that the kernel
// before it (which writes no cell the gathers read) saved the snapshots:
// each of its CTAs saves its own block's, after its own writes.
struct FillPass {
  GhostSeg seg[kMaxSeg];
  int nseg;             // 0: no fill
  int groups;           // groups of variables over the segments (row_groups)
  int tile_seg;         // segment mirrored in the consuming kernel's shared memory (-1: none)
  double *snapbuf;      // [nseg][nsnaps][8], values of the segment's type (snap_rows)
};
struct FillFuse {
  const GhostOp *ops;
  const GhostSnap *snaps;
  int nsnaps;           // snapshot rows per segment in a buffer
  FillPass apply;       // the fill this kernel consumes: gathered into the CTA's block first
  FillPass save;        // the next fill: the CTA's block's snapshots, saved last
};

// A thread's share of a fill is one gather (or snapshot) and a group of
// consecutive variables of one segment, 4 of a float field (which all have 8
// variables) or 2 of a double one: the gather is read once, and the values'
// loads, at constant distances, are in flight together.  The fills wait on the
// latency of two dependent loads (gather, value): with a variable per thread,
// 13 rounds of it per block and fill of B, ff and gg for a CTA of 128; with
// groups, 4 (FP32) or 7.  More per thread costs registers, and with them the
// resident warps that hide the same latency in large batches.
template <typename F> __host__ __device__ constexpr int row_group() { return sizeof(F) == 4 ? 4 : 2; }
__host__ __device__ constexpr int row_groups(int nv, int f32) { return f32 ? nv / 4 : (nv + 1) / 2; }

// segment q and first variable k0 of group g
__device__ __forceinline__ GhostSeg pass_seg(const FillPass &p, int g, int &q, int &k0) {
  GhostSeg s = p.seg[0];
  q = 0;
  if (p.nseg > 1 && g >= row_groups(s.nv, s.f32)) { g -= row_groups(s.nv, s.f32); s = p.seg[1]; q = 1; }
  if (p.nseg > 2 && q == 1 && g >= row_groups(s.nv, s.f32)) { g -= row_groups(s.nv, s.f32); s = p.seg[2]; q = 2; }
  k0 = g * (s.f32 ? 4 : 2);
  return s;
}

// a group of variables from k0 on of one gather: a, and b for a pair's second cell
template <typename F>
struct GhostVals {
  F a[row_group<F>()], b[row_group<F>()];
};

template <int N, typename F>
__device__ __forceinline__ void ghost_load(const GhostSeg &s, const GhostOp &op, int k0, const F *snap,
                                           GhostVals<F> &v) {
  constexpr int NN = N * N;
  const F *c = static_cast<const F *>(s.field) + (static_cast<size_t>(op.src_slot) * s.nv + k0) * NN + op.src_pos;
  const int left = sizeof(F) == 4 ? 4 : s.nv - k0;
  if (op.type == GOP_COPY2) {  // even positions in an even-sized plane: aligned pairs
    using P2 = typename std::conditional<sizeof(F) == 4, float2, double2>::type;
#pragma unroll
    for (int j = 0; j < row_group<F>(); j++)
      if (j < left) {
        const P2 x = *reinterpret_cast<const P2 *>(c + j * NN);
        v.a[j] = x.x;
        v.b[j] = x.y;
      }
    return;
  }
  if (op.type == GOP_COPY) {
#pragma unroll
    for (int j = 0; j < row_group<F>(); j++)
      if (j < left) v.a[j] = c[j * NN];
    return;
  }
  if (op.type == GOP_FINE) {
#pragma unroll
    for (int j = 0; j < row_group<F>(); j++)
      if (j < left) {
        const F *x = c + j * NN;
        v.a[j] = fine_value<F>(s.kind, k0 + j, x[0], x[N], x[1], x[1 + N]);
      }
    return;
  }
  const F *r = snap + static_cast<size_t>(op.src_slot) * 8 + k0;
#pragma unroll
  for (int j = 0; j < row_group<F>(); j++)
    if (j < left)
      v.a[j] = op.type == GOP_SNAP ? r[j] : fine_value<F>(s.kind, k0 + j, r[j], r[8 + j], r[16 + j], r[24 + j]);
}

template <int N, typename F>
__device__ __forceinline__ void ghost_store(const GhostSeg &s, const GhostOp &op, int k0, const GhostVals<F> &v,
                                            F *tile) {
  constexpr int NN = N * N;
  F *d = static_cast<F *>(s.field) + (static_cast<size_t>(op.dst_slot) * s.nv + k0) * NN + op.dst_pos;
  F *tl = tile + k0 * NN + op.dst_pos;
  const int left = sizeof(F) == 4 ? 4 : s.nv - k0;
  if (op.type == GOP_COPY2) {
    using P2 = typename std::conditional<sizeof(F) == 4, float2, double2>::type;
#pragma unroll
    for (int j = 0; j < row_group<F>(); j++)
      if (j < left) {
        P2 x;
        x.x = v.a[j];
        x.y = v.b[j];
        *reinterpret_cast<P2 *>(d + j * NN) = x;
        if (tile) *reinterpret_cast<P2 *>(tl + j * NN) = x;
      }
    return;
  }
#pragma unroll
  for (int j = 0; j < row_group<F>(); j++)
    if (j < left) {
      d[j * NN] = v.a[j];
      if (tile) tl[j * NN] = v.a[j];
    }
}

// threadIdx.x, opaque to the compiler: in a kernel that loops over blocks it
// would otherwise compute every index that depends on the thread once, before
// the loop, and spill them (0.5 KB per thread in k_stage_dyn).
__device__ __forceinline__ int block_tid() {
  int t = threadIdx.x;
  asm volatile("" : "+r"(t));
  return t;
}

// item e of the fill `f.apply` on the block of task t, n gathers per group.
// S is the storage type of the bulk fields: FP64 handles have no float field.
template <int N, typename S>
__device__ __forceinline__ void fill_item(const FillFuse &f, const LeafTask &t, int e, int n, S *tile) {
  const int g = e / n;
  const GhostOp op = f.ops[t.op_begin + (e - g * n)];
  int q, k0;
  const GhostSeg s = pass_seg(f.apply, g, q, k0);
  S *tl = q == f.apply.tile_seg ? tile : nullptr;
  if (sizeof(S) == 4 && s.f32) {
    GhostVals<float> v;
    ghost_load<N, float>(s, op, k0, snap_rows<float>(f.apply.snapbuf, q, f.nsnaps), v);
    ghost_store<N, float>(s, op, k0, v, reinterpret_cast<float *>(tl));
  } else {
    GhostVals<double> v;
    ghost_load<N, double>(s, op, k0, snap_rows<double>(f.apply.snapbuf, q, f.nsnaps), v);
    ghost_store<N, double>(s, op, k0, v, sizeof(S) == 8 ? reinterpret_cast<double *>(tl) : nullptr);
  }
}

// the gathers of the fill `f.apply` into the ghost cells of task t's block
// (consecutive threads take consecutive gathers); the caller synchronises
// the CTA afterwards
template <int N, typename S>
__device__ __forceinline__ void fill_apply_task(const FillFuse &f, const LeafTask &t, int tid, int nthr) {
  const int n = t.op_count, total = n * f.apply.groups;
#pragma unroll 1
  for (int e = tid; e < total; e += nthr) fill_item<N, S>(f, t, e, n, static_cast<S *>(nullptr));
}

// The first item of a thread, loaded ahead (while the fused stage kernel's
// bulk copy is in flight) if it is of the staged field, segment 0 (of the
// storage type), and stored by fill_apply_task_after.
template <typename S>
struct FillPre {
  GhostOp op;
  GhostVals<S> v;
  int k0;
  bool on;
};

template <int N, typename S>
__device__ __forceinline__ void fill_prefetch(const FillFuse &f, const LeafTask &t, int tid, FillPre<S> &p) {
  const int n = t.op_count, g = n > 0 ? tid / n : 0;
  p.on = f.apply.nseg != 0 && n > 0 && g < row_groups(f.apply.seg[0].nv, f.apply.seg[0].f32);
  if (!p.on) return;
  p.op = f.ops[t.op_begin + (tid - g * n)];
  p.k0 = g * row_group<S>();
  ghost_load<N, S>(f.apply.seg[0], p.op, p.k0, snap_rows<S>(f.apply.snapbuf, 0, f.nsnaps), p.v);
}

// fill_apply_task, `tile` the staged copy, with what `p` holds already loaded
template <int N, typename S>
__device__ __forceinline__ void fill_apply_task_after(const FillFuse &f, const LeafTask &t, int tid, int nthr, S *tile,
                                                      const FillPre<S> &p) {
  if (p.on) ghost_store<N, S>(f.apply.seg[0], p.op, p.k0, p.v, tile);
  const int n = t.op_count, total = n * f.apply.groups;
#pragma unroll 1
  for (int e = p.on ? tid + nthr : tid; e < total; e += nthr) fill_item<N, S>(f, t, e, n, tile);
}

// a group of variables from k0 on of a snapshot
template <int NN, typename F>
__device__ __forceinline__ void snap_vals(const GhostSeg &s, const GhostSnap &sn, int k0, F *row) {
  const F *c = static_cast<const F *>(s.field) + (static_cast<size_t>(sn.slot) * s.nv + k0) * NN + sn.pos;
  const int left = sizeof(F) == 4 ? 4 : s.nv - k0;
  F v[row_group<F>()];
#pragma unroll
  for (int j = 0; j < row_group<F>(); j++)
    if (j < left) v[j] = c[j * NN];
#pragma unroll
  for (int j = 0; j < row_group<F>(); j++)
    if (j < left) row[k0 + j] = v[j];
}
template <int NN, typename S>
__device__ __forceinline__ void snap_one(const FillFuse &f, const GhostSnap &sn, int r, int g) {
  int q, k0;
  const GhostSeg s = pass_seg(f.save, g, q, k0);
  const size_t to = static_cast<size_t>(r) * 8;
  if (sizeof(S) == 4 && s.f32) snap_vals<NN, float>(s, sn, k0, snap_rows<float>(f.save.snapbuf, q, f.nsnaps) + to);
  else snap_vals<NN, double>(s, sn, k0, snap_rows<double>(f.save.snapbuf, q, f.nsnaps) + to);
}

// the snapshots of the next fill (`f.save`) that lie in task t's block; the
// caller synchronises the CTA before, after its own writes to the fields
template <int N, typename S>
__device__ __forceinline__ void fill_save_task(const FillFuse &f, const LeafTask &t, int tid, int nthr) {
  const int n = t.snap_count, total = n * f.save.groups;
#pragma unroll 1
  for (int e = tid; e < total; e += nthr) {
    const int g = e / n, r = t.snap_begin + (e - g * n);
    snap_one<N * N, S>(f, f.snaps[r], r, g);
  }
}

// every snapshot of the next fill, from any thread of the grid: for a
// kernel that writes none of the saved fields
template <int N, typename S>
__device__ __forceinline__ void fill_save_all(const FillFuse &f, size_t gtid, size_t gsize) {
  const size_t total = static_cast<size_t>(f.nsnaps) * f.save.groups;
#pragma unroll 1
  for (size_t e = gtid; e < total; e += gsize) {
    const int g = static_cast<int>(e / f.nsnaps);
    const int r = static_cast<int>(e - static_cast<size_t>(g) * f.nsnaps);
    const GhostSnap sn = f.snaps[r];
    if (sn.slot >= 0) snap_one<N * N, S>(f, sn, r, g);
  }
}

}  // namespace amr
