// Device bodies of the halo, restriction and reflux ops: one op over the NT threads of a
// block. The standalone op kernels launch one op per block; the op program
// (program.cu) runs them inside one launch.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "halo.cuh"
#include "layout.cuh"

namespace wb {

// A thread's place among the NT threads that run one op (a whole block, or one warp of it).
template <int NT>
__device__ __forceinline__ unsigned op_lane() {
  return threadIdx.x % unsigned(NT);
}

// element offset of haloed index (i, j, k) of a patch (k ignored in 2D)
__device__ __forceinline__ int64_t offset_of(const PatchDesc& P, int i, int j, int k) {
  if (P.pitch1) return int64_t(i) * P.pitch0 + int64_t(j) * P.pitch1 + k;
  return int64_t(i) * P.pitch0 + j;
}

// the same from the pitches
__device__ __forceinline__ int64_t pitched(int64_t pitch0, int64_t pitch1, int i, int j, int k) {
  return pitch1 ? i * pitch0 + j * pitch1 + k : i * pitch0 + j;
}

constexpr int kOpThreads = 64;  // threads of the block that runs one op

// Fields [lo, lo + NF) of one copied point (NF a compile-time count, or 0: nf of them, at
// most 8): every field's value first, then the stores (an op never writes a point it reads).
template <typename S, int NF>
__device__ __forceinline__ void copy_fields(S* __restrict__ pool, const CopyOp& op, int64_t od, int64_t fd, int64_t o1,
                                            int64_t f1, int64_t o2, int64_t f2) {
  constexpr int kMost = NF ? NF : 8;
  const int nf = NF ? NF : op.field_hi - op.field_lo;
  const bool plain = op.w1 == 1.0 && op.w2 == 0.0 && op.negate < 0;
  S v[kMost];
#pragma unroll
  for (int f = 0; f < kMost; ++f)
    if (f < nf) v[f] = pool[o1 + f * f1];
  if (!plain) {  // uniform over the op
#pragma unroll
    for (int f = 0; f < kMost; ++f) {
      if (f >= nf) continue;
      S x = S(op.w1) * v[f];
      if (op.w2 != 0.0) x += S(op.w2) * pool[o2 + f * f2];
      v[f] = op.field_lo + f == op.negate ? -x : x;
    }
  }
#pragma unroll
  for (int f = 0; f < kMost; ++f)
    if (f < nf) pool[od + f * fd] = v[f];
}

// The points of one copy op, over the NT threads of the block. The field counts of the two
// layouts (cells: 6 in 2D, 5 in 3D; potentials: 1) have code of their own: with the general
// eight guarded fields most of a one-field op's instructions do nothing.
template <typename S, int NT = kOpThreads>
__device__ __forceinline__ void copy_op(S* __restrict__ pool, const PatchDesc* __restrict__ patches, const CopyOp& op) {
  const PatchDesc& D = patches[op.dst];
  const PatchDesc& A = patches[op.src1];
  const PatchDesc& B = patches[op.src2 >= 0 ? op.src2 : op.src1];
  const int64_t fd = D.fstride, f1 = A.fstride, f2 = B.fstride;
  const int64_t bd = D.off + op.field_lo * fd, b1 = A.off + op.field_lo * f1, b2 = B.off + op.field_lo * f2;
  const int64_t d0 = D.pitch0, d1 = D.pitch1, a0 = A.pitch0, a1 = A.pitch1, c0 = B.pitch0, c1 = B.pitch1;
  const bool two = op.w2 != 0.0;
  // 32-bit point index (the host keeps every op below 2^31 points)
  const unsigned n1 = unsigned(op.n[1]), n2 = unsigned(op.n[2]);
  const unsigned count = unsigned(op.n[0]) * n1 * n2;
  for (unsigned t = op_lane<NT>(); t < count; t += NT) {
    const unsigned line = t / n2;
    const int p2 = int(t - line * n2);
    const int p0 = int(line / n1);
    const int p1 = int(line - unsigned(p0) * n1);
    const int64_t od = bd + pitched(d0, d1, op.d[0] + p0, op.d[1] + p1, op.d[2] + p2);
    const int64_t o1 = b1 + pitched(a0, a1, op.s1[0] + op.m1[0] * p0, op.s1[1] + op.m1[1] * p1, op.s1[2] + op.m1[2] * p2);
    const int64_t o2 =
        two ? b2 + pitched(c0, c1, op.s2[0] + op.m2[0] * p0, op.s2[1] + op.m2[1] * p1, op.s2[2] + op.m2[2] * p2) : 0;
    switch (op.field_hi - op.field_lo) {
      case 1: copy_fields<S, 1>(pool, op, od, fd, o1, f1, o2, f2); break;
      case 5: copy_fields<S, 5>(pool, op, od, fd, o1, f1, o2, f2); break;
      case 6: copy_fields<S, 6>(pool, op, od, fd, o1, f1, o2, f2); break;
      default: copy_fields<S, 0>(pool, op, od, fd, o1, f1, o2, f2); break;
    }
  }
}

// A plain copy (w1 = 1, no second source, nothing negated) of NF fields of up to two points:
// all loads before the stores.
template <typename S, int NF>
__device__ __forceinline__ void copy_two(S* __restrict__ pool, bool both, int64_t d0, int64_t d1, int64_t fd, int64_t s0,
                                         int64_t s1, int64_t fs) {
  S v[2][NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    v[0][f] = pool[s0 + f * fs];
    if (both) v[1][f] = pool[s1 + f * fs];
  }
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    pool[d0 + f * fd] = v[0][f];
    if (both) pool[d1 + f * fd] = v[1][f];
  }
}

// The points of one copy op, two per thread and pass where it is a plain copy (an op never
// writes a point it reads): for the standalone copy launches, whose ops are large where the
// lists are (a big box's halos). Other copies go as copy_op. B200, a fill: 256^3 float32 54 ->
// 45 us, 150 x 97 x 75 float64 17.1 -> 13.8 us, 512 planes 53 -> 34 us.
template <typename S, int NT = kOpThreads>
__device__ __forceinline__ void copy_op_pairs(S* __restrict__ pool, const PatchDesc* __restrict__ patches,
                                              const CopyOp& op) {
  const int nf = op.field_hi - op.field_lo;
  if (!(op.w1 == 1.0 && op.w2 == 0.0 && op.negate < 0) || (nf != 1 && nf != 5 && nf != 6)) {
    copy_op<S, NT>(pool, patches, op);
    return;
  }
  const PatchDesc& D = patches[op.dst];
  const PatchDesc& A = patches[op.src1];
  const int64_t fd = D.fstride, fs = A.fstride;
  const int64_t bd = D.off + op.field_lo * fd, bs = A.off + op.field_lo * fs;
  const int64_t dp0 = D.pitch0, dp1 = D.pitch1, sp0 = A.pitch0, sp1 = A.pitch1;
  // 32-bit point index (the host keeps every op below 2^31 points)
  const unsigned n1 = unsigned(op.n[1]), n2 = unsigned(op.n[2]);
  const unsigned count = unsigned(op.n[0]) * n1 * n2;
  for (unsigned t0 = op_lane<NT>(); t0 < count; t0 += 2 * NT) {
    int64_t d[2], s[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const unsigned t = min(t0 + u * NT, count - 1);
      const unsigned line = t / n2;
      const int p2 = int(t - line * n2);
      const int p0 = int(line / n1);
      const int p1 = int(line - unsigned(p0) * n1);
      d[u] = bd + pitched(dp0, dp1, op.d[0] + p0, op.d[1] + p1, op.d[2] + p2);
      s[u] = bs + pitched(sp0, sp1, op.s1[0] + op.m1[0] * p0, op.s1[1] + op.m1[1] * p1, op.s1[2] + op.m1[2] * p2);
    }
    const bool both = t0 + NT < count;
    if (nf == 1)
      copy_two<S, 1>(pool, both, d[0], d[1], fd, s[0], s[1], fs);
    else if (nf == 5)
      copy_two<S, 5>(pool, both, d[0], d[1], fd, s[0], s[1], fs);
    else
      copy_two<S, 6>(pool, both, d[0], d[1], fd, s[0], s[1], fs);
  }
}

// Fine halo points from the coarse patch below. Fine haloed index f along an axis
// corresponds to level index g = f - 2 + box_lo; the coarse level index is g / 2.
template <typename S>
__device__ __forceinline__ void axis_weights(int node_axis, int g, int& c0, int& cnt, S (&w)[4]) {
  // returns coarse level indices c0 .. c0+cnt-1 with weights w
  if (node_axis) {
    if ((g & 1) == 0) {
      c0 = g >> 1;
      cnt = 1;
      w[0] = S(1);
    } else {
      c0 = (g >> 1) - 1;  // floor for negative g too (arithmetic shift)
      cnt = 4;
      w[0] = S(-1.0 / 16);
      w[1] = S(9.0 / 16);
      w[2] = S(9.0 / 16);
      w[3] = S(-1.0 / 16);
    }
  } else {
    const int c = g >> 1;
    if ((g & 1) == 0) {
      c0 = c - 1;
      w[0] = S(0.25);
      w[1] = S(0.75);
    } else {
      c0 = c;
      w[0] = S(0.75);
      w[1] = S(0.25);
    }
    cnt = 2;
  }
}

// NF cell-centred fields of one fine point: two coarse cells along every axis, all loads of
// all fields before the stores; each field's terms in the order a0, a1, a2.
template <typename S, int NDIM, int NF>
__device__ __forceinline__ void interp_cells(const S* coarse, int64_t cf, int64_t cp0, int64_t cp1,
                                             const S (&w)[3][4], S* out, int64_t ff) {
  S acc[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) acc[f] = S(0);
#pragma unroll 1
  for (int a0 = 0; a0 < 2; ++a0)
#pragma unroll
    for (int a1 = 0; a1 < 2; ++a1)
#pragma unroll
      for (int a2 = 0; a2 < (NDIM == 3 ? 2 : 1); ++a2) {
        const S wt = (a0 == 0 ? w[0][0] : w[0][1]) * w[1][a1] * w[2][a2];
        const S* c = coarse + a0 * cp0 + (NDIM == 3 ? a1 * cp1 + a2 : a1);
#pragma unroll
        for (int f = 0; f < NF; ++f) acc[f] += wt * c[f * cf];
      }
#pragma unroll
  for (int f = 0; f < NF; ++f) out[f * ff] = acc[f];
}

// One field of one fine point, any mix of node and cell axes (1, 2 or 4 coarse points along
// an axis), terms in the order a0, a1, a2; the points of one a0 are loaded together.
template <typename S, int NDIM>
__device__ __forceinline__ S interp_value(const S* coarse, int64_t cp0, int64_t cp1, const int (&cnt)[3],
                                          const S (&w)[3][4]) {
  constexpr int K2 = NDIM == 3 ? 4 : 1;
  S acc = S(0);
#pragma unroll 1
  for (int a0 = 0; a0 < cnt[0]; ++a0) {
    const S w0 = a0 == 0 ? w[0][0] : (a0 == 1 ? w[0][1] : (a0 == 2 ? w[0][2] : w[0][3]));
    S v[4][K2];
#pragma unroll
    for (int a1 = 0; a1 < 4; ++a1)
#pragma unroll
      for (int a2 = 0; a2 < K2; ++a2)
        if (a1 < cnt[1] && a2 < cnt[2]) v[a1][a2] = coarse[a0 * cp0 + (NDIM == 3 ? a1 * cp1 + a2 : a1)];
#pragma unroll
    for (int a1 = 0; a1 < 4; ++a1)
#pragma unroll
      for (int a2 = 0; a2 < K2; ++a2)
        if (a1 < cnt[1] && a2 < cnt[2]) acc += w0 * w[1][a1] * w[2][a2] * v[a1][a2];
  }
  return acc;
}

// The points of one interpolation op, over the NT threads of the block. The cell fields of
// the layouts take two weights an axis and all fields at once; node-centred fields (the
// potentials, one field an op) take up to 4 x 4 x 2 points of their one field. Guarding eight
// fields at every one of 64 weights, as one code for both would, is ~800 issue slots a point
// and 86 registers; here 64 (16 blocks an SM). B200, a level's fill (interpolation and
// copies): 3D, 592,000 + 938,000 points 212 -> 30 us; 2D, 12,000 + 148,000 points 13 -> 6 us.
template <typename S, int NDIM, int NT>
__device__ __forceinline__ void interp_points(S* __restrict__ pool, const PatchDesc* __restrict__ patches,
                                              const InterpOp& op) {
  const PatchDesc& F = patches[op.fine];
  const PatchDesc& C = patches[op.coarse];
  const int64_t cf = C.fstride, cp0 = C.pitch0, cp1 = C.pitch1, ff = F.fstride, fp0 = F.pitch0, fp1 = F.pitch1;
  const S* cbase = pool + C.off;
  S* fbase = pool + F.off;
  const int lo = op.field_lo, nf = op.field_hi - op.field_lo;
  // 32-bit point index (the host keeps every op below 2^31 points)
  const unsigned n1 = unsigned(op.n[1]), n2 = unsigned(op.n[2]);
  const unsigned count = unsigned(op.n[0]) * n1 * n2;
  for (unsigned t = op_lane<NT>(); t < count; t += NT) {
    const unsigned line = t / n2;
    const int q0 = int(line / n1);
    const int q[3] = {q0, int(line - unsigned(q0) * n1), int(t - line * n2)};
    int c0[3] = {0, 0, 0}, cnt[3] = {1, 1, 1};
    S w[3][4];
    w[2][0] = S(1);
#pragma unroll
    for (int a = 0; a < NDIM; ++a) {
      const int g = op.d[a] + q[a] - kHalo + op.fine_lo[a];  // fine level index
      axis_weights<S>((op.node_mask >> a) & 1, g, c0[a], cnt[a], w[a]);
      c0[a] = c0[a] - op.coarse_lo[a] + kHalo;  // coarse haloed index
    }
    const S* c = cbase + lo * cf + pitched(cp0, NDIM == 3 ? cp1 : 0, c0[0], c0[1], c0[2]);
    S* out = fbase + lo * ff + pitched(fp0, NDIM == 3 ? fp1 : 0, op.d[0] + q[0], op.d[1] + q[1], op.d[2] + q[2]);
    if (op.node_mask == 0 && nf == (NDIM == 3 ? 5 : 6)) {
      interp_cells<S, NDIM, NDIM == 3 ? 5 : 6>(c, cf, cp0, cp1, w, out, ff);
    } else {
#pragma unroll 1
      for (int f = 0; f < nf; ++f) out[f * ff] = interp_value<S, NDIM>(c + f * cf, cp0, cp1, cnt, w);
    }
  }
}

template <typename S, int NT = kOpThreads>
__device__ __forceinline__ void interp_op(S* __restrict__ pool, const PatchDesc* __restrict__ patches,
                                          const InterpOp& op) {
  if (op.ndim == 3)
    interp_points<S, 3, NT>(pool, patches, op);
  else
    interp_points<S, 2, NT>(pool, patches, op);
}

// The coarse points of one restriction op, over the NT threads of the block: the mean of
// the fine values along cell-centred axes, the coincident fine value along node axes.
template <typename S, int NT = kOpThreads>
__device__ __forceinline__ void restrict_op(S* __restrict__ pool, const PatchDesc* __restrict__ patches,
                                            const RestrictOp& op) {
  const PatchDesc F = patches[op.fine];
  const PatchDesc C = patches[op.coarse];
  int cnt[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) cnt[a] = (a < op.ndim && !((op.node_mask >> a) & 1)) ? 2 : 1;
  const int total = cnt[0] * cnt[1] * cnt[2];
  const S scale = S(1) / S(total);
  const int lo = op.field_lo, hi = op.field_hi;
  // 32-bit point index (the host keeps every op below 2^31 points)
  const unsigned n1 = unsigned(op.n[1]), n2 = unsigned(op.n[2]);
  const unsigned count = unsigned(op.n[0]) * n1 * n2;
  for (unsigned t = op_lane<NT>(); t < count; t += NT) {
    const unsigned line = t / n2;
    const int q2 = int(t - line * n2);
    const int q1 = int(line % n1);
    const int q0 = int(line / n1);
    const int ci[3] = {op.c[0] + q0, op.c[1] + q1, op.c[2] + q2};  // coarse haloed
    const int fi[3] = {op.f[0] + 2 * q0, op.f[1] + 2 * q1, op.f[2] + 2 * q2};  // fine haloed start
    // every fine value of every field first (fields innermost; each field's terms in the
    // order a0, a1, a2), then the stores
    S acc[8];
#pragma unroll
    for (int f = 0; f < 8; ++f) acc[f] = S(0);
#pragma unroll
    for (int a0 = 0; a0 < 2; ++a0)
#pragma unroll
      for (int a1 = 0; a1 < 2; ++a1)
#pragma unroll
        for (int a2 = 0; a2 < 2; ++a2) {
          if (a0 < cnt[0] && a1 < cnt[1] && a2 < cnt[2]) {
            const S* ff = pool + F.off + offset_of(F, fi[0] + a0, fi[1] + a1, op.ndim == 3 ? fi[2] + a2 : 0);
#pragma unroll
            for (int f = 0; f < 8; ++f)
              if (f >= lo && f < hi) acc[f] += ff[f * F.fstride];
          }
        }
    S* out = pool + C.off + offset_of(C, ci[0], ci[1], op.ndim == 3 ? ci[2] : 0);
#pragma unroll
    for (int f = 0; f < 8; ++f)
      if (f >= lo && f < hi) out[f * C.fstride] = total == 1 ? acc[f] : acc[f] * scale;
  }
}

// Apply the register of one interface to the coarse cells beside it, then clear it:
// U -= sign * (0.5 dt) * reg / dx (sign +1 where the interface is the cell's upper face).
// The ops run together must touch disjoint cells (no atomics).
template <typename S, int NT>
__device__ __forceinline__ void reflux_op(S* __restrict__ pool, const PatchDesc* __restrict__ patches,
                                          const RefluxOp& op, double* __restrict__ reg,
                                          const double* dt) {
  const PatchDesc C = patches[op.coarse];
  const double scale = 0.5 * dt[C.instance];
  const int64_t count = int64_t(op.len) * op.ncomp;
  for (int64_t t = op_lane<NT>(); t < count; t += NT) {
    const int q = int(t / op.len), s = int(t % op.len);
    const int s1 = s / op.width, s2 = s % op.width;
    int idx[3] = {op.c[0], op.c[1], op.c[2]};
    idx[op.t1] += s1;
    if (op.t2 >= 0) idx[op.t2] += s2;
    const int64_t o = offset_of(C, idx[0], idx[1], idx[2]);
    double& r = reg[op.reg_off + int64_t(q) * op.len + s];
    S* u = pool + C.off + int64_t(op.field[q]) * C.fstride + o;
    *u = S(double(*u) - op.sign * scale * r / op.dx);
    r = 0.0;
  }
}

}  // namespace wb
