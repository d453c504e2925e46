// Device bodies of the stable-time-step reduction (carafe/kernels/mhd_rate/mhd_rate_pyccel.py:30-83
// in 2D, carafe/mhd3d.py:674-724 in 3D; dt as carafe/mhd.py:930-963): one chunk of cells
// over the threads of a block, and the step of one instance. Shared by the rate kernels
// and the op program.
#pragma once

#include "layout.cuh"
#include "numerics.cuh"
#include "wb_internal.cuh"

namespace wb {

// Cells per work item of the rate reduction (the host cuts every patch into such chunks).
constexpr unsigned kRateChunk = 2048;

__device__ __forceinline__ unsigned long long rate_min_identity() {
  return double_to_key(__longlong_as_double(0x7ff0000000000000ll));
}

// Where a rate block reduces: the instance's key pair and, optionally, the density-minimum
// key of the patch's level. A patch whose instance or level lies outside the key arrays
// is skipped (its block reduces nothing) and flagged in `error` (nullable).
struct RateSlots {
  unsigned long long* keys;        // [2 * ninstances]
  int ninstances;
  unsigned long long* level_keys;  // [ninstances * nlevels] or null
  int nlevels;
  unsigned* error;                 // nullable
};

__device__ __forceinline__ bool rate_slot(const PatchDesc& P, const RateSlots& r, unsigned long long** keys,
                                          unsigned long long** level_min) {
  const bool ok = P.instance >= 0 && P.instance < r.ninstances && (!r.level_keys || (P.level >= 0 && P.level < r.nlevels));
  if (!ok) {
    if (r.error && threadIdx.x == 0) atomicOr(r.error, 1u);
    return false;
  }
  *keys = r.keys + 2 * P.instance;
  *level_min = r.level_keys ? r.level_keys + P.instance * r.nlevels + P.level : nullptr;
  return true;
}

// The rate's arithmetic with every rounding written out, so that each kernel that forms a
// cell's rate (one launch or several, any unrolling) gets the same bits: left to the
// compiler, the choice which product of a sum to fuse differed between instantiations in
// one cell of twenty.
template <typename S>
struct RateMath;

template <>
struct RateMath<float> {
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
  static __device__ __forceinline__ float div(float a, float, float inv_b) { return __fmul_rn(a, inv_b); }
  static __device__ __forceinline__ float quotient(float a, float b, float inv_b) { return div(a, b, inv_b); }
  // a / b + c and a / h - b / k
  static __device__ __forceinline__ float div_plus(float a, float, float inv_b, float c) { return __fmaf_rn(a, inv_b, c); }
  static __device__ __forceinline__ float ratio_plus(float a, float b, float inv_b, float c) { return div_plus(a, b, inv_b, c); }
  static __device__ __forceinline__ float curl(float a, float, float ih, float b, float, float ik) {
    return __fmaf_rn(a, ih, -__fmul_rn(b, ik));
  }
  static __device__ __forceinline__ float sqrt(float x) {
    return x > 0.0f ? __fmul_rn(x, rsqrtf(x)) : 0.0f;
  }
};

template <>
struct RateMath<double> {
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double fma(double a, double b, double c) { return __fma_rn(a, b, c); }
  static __device__ __forceinline__ double div(double a, double b, double inv_b) { return Math<double>::div(a, b, inv_b); }
  // a / b also where a is infinite: a signal speed without bound gives no step, not a NaN that
  // the maximum passes over
  static __device__ __forceinline__ double quotient(double a, double b, double inv_b) { return MathIeee::div(a, b, inv_b); }
  static __device__ __forceinline__ double div_plus(double a, double b, double inv_b, double c) {
    return __dadd_rn(div(a, b, inv_b), c);
  }
  static __device__ __forceinline__ double ratio_plus(double a, double b, double inv_b, double c) {
    return __dadd_rn(quotient(a, b, inv_b), c);
  }
  static __device__ __forceinline__ double curl(double a, double h, double ih, double b, double k, double ik) {
    return __dadd_rn(div(a, h, ih), -div(b, k, ik));
  }
  static __device__ __forceinline__ double sqrt(double x) { return x > 0.0 ? ::sqrt(x) : 0.0; }
};

// Fast magnetosonic speed from a2 = gamma p / rho, the normal field and the field squared.
template <typename S, int NDIM>
__device__ __forceinline__ S rate_speed(S a2, S bn, S field2, S rho, S inv_rho) {
  using Q = RateMath<S>;
  const S s = Q::div_plus(field2, rho, inv_rho, a2);
  const S y = Q::mul(Q::mul(Q::mul(S(4), a2), bn), bn);
  const S disc = NDIM == 2 ? Q::div_plus(-y, rho, inv_rho, Q::mul(s, s)) : Q::fma(s, s, -Q::div(y, rho, inv_rho));
  const S root = disc > S(0) ? Q::sqrt(disc) : S(0);
  return Q::sqrt(Q::mul(S(0.5), Q::add(s, root)));
}

// (gamma - 1) (E - rho v^2 / 2 - B^2 / 2)
template <typename S>
__device__ __forceinline__ S rate_pressure(S gm1, S e, S rho, S u, S v, S w, S field2) {
  using Q = RateMath<S>;
  const S v2 = Q::fma(w, w, Q::fma(u, u, Q::mul(v, v)));
  const S rest = Q::fma(-Q::mul(S(0.5), rho), v2, e);
  return Q::mul(gm1, Q::add(rest, -Q::mul(S(0.5), field2)));
}

// Largest signal rate and smallest density of the cells begin + thread, begin + thread + NT,
// ... (`rounds` of them, those inside the patch). Issue and latency bound (~200 instructions
// a float32 3D cell against 32 bytes); unrolling by two raises the registers and loses warps.
// 2D:
template <typename S, int NT>
__device__ __forceinline__ void rate_cells2d(const S* src, const PatchDesc& P, unsigned begin, int rounds,
                                             double b0x, double b0y, double gamma, S& largest, S& smallest) {
  const int64_t pitch = P.pitch0, fs = P.fstride;
  using M = Math<S>;
  using Q = RateMath<S>;
  const S dx = S(P.dx[0]), dy = S(P.dx[1]);
  const S idx = M::inv(dx), idy = M::inv(dy);
  const S g = S(gamma), gm1 = g - S(1), bx0 = S(b0x), by0 = S(b0y);
  // work-list indices are 32-bit (chunk_start is int): 32-bit index arithmetic
  const int ny = P.n[1];
  const unsigned total = unsigned(P.n[0]) * unsigned(ny);
#pragma unroll 1
  for (int s = 0; s < rounds; ++s) {
    const unsigned t = begin + unsigned(s) * NT + threadIdx.x;
    if (t >= total) continue;
    const unsigned row = t / unsigned(ny);
    const int i = int(row) + kHalo, j = int(t - row * unsigned(ny)) + kHalo;
    const int64_t c = int64_t(i) * pitch + j;
    const S* A = src + 6 * fs;
    const S a00 = A[c], a01 = A[c + 1], a10 = A[c + pitch], a11 = A[c + pitch + 1];
    const S r = src[c];
    const S ir = M::inv(r);
    const S u = Q::div(src[fs + c], r, ir), v = Q::div(src[2 * fs + c], r, ir), w = Q::div(src[3 * fs + c], r, ir);
    const S bz = src[5 * fs + c], e = src[4 * fs + c];
    const S bx = Q::mul(S(0.5), Q::add(Q::div_plus(a01 - a00, dy, idy, bx0), Q::div_plus(a11 - a10, dy, idy, bx0)));
    const S by = Q::mul(S(0.5), Q::add(Q::div_plus(a00 - a10, dx, idx, by0), Q::div_plus(a01 - a11, dx, idx, by0)));
    const S b2 = Q::fma(bz, bz, Q::fma(bx, bx, Q::mul(by, by)));
    const S p = rate_pressure(gm1, e, r, u, v, w, b2);
    const S a2 = Q::quotient(Q::mul(g, p), r, ir);
    const S cx = Q::add(rabs(u), rate_speed<S, 2>(a2, bx, b2, r, ir));
    const S cy = Q::add(rabs(v), rate_speed<S, 2>(a2, by, b2, r, ir));
    largest = rmax(largest, Q::ratio_plus(cx, dx, idx, Q::quotient(cy, dy, idy)));
    smallest = rmin(smallest, r);
  }
}

// 3D:
template <typename S, int NT>
__device__ __forceinline__ void rate_cells3d(const S* src, const PatchDesc& P, unsigned begin, int rounds,
                                             double b0x, double b0y, double b0z, double gamma, S& largest, S& smallest) {
  const int64_t p0 = P.pitch0, p1 = P.pitch1, fs = P.fstride;
  using M = Math<S>;
  using Q = RateMath<S>;
  const S dx = S(P.dx[0]), dy = S(P.dx[1]), dz = S(P.dx[2]);
  const S idx = M::inv(dx), idy = M::inv(dy), idz = M::inv(dz);
  const S g = S(gamma), gm1 = g - S(1);
  // work-list indices are 32-bit (chunk_start is int): 32-bit index arithmetic
  const int ny = P.n[1], nz = P.n[2];
  const unsigned total = unsigned(P.n[0]) * unsigned(ny) * unsigned(nz);
#pragma unroll 1
  for (int s = 0; s < rounds; ++s) {
    const unsigned t = begin + unsigned(s) * NT + threadIdx.x;
    if (t >= total) continue;
    const unsigned line = t / unsigned(nz);
    const unsigned plane = line / unsigned(ny);
    const int i = int(plane) + kHalo;
    const int j = int(line - plane * unsigned(ny)) + kHalo;
    const int k = int(t - line * unsigned(nz)) + kHalo;
    const int64_t o = int64_t(i) * p0 + int64_t(j) * p1 + k;
    const S* Ax = src + 5 * fs;
    const S* Ay = src + 6 * fs;
    const S* Az = src + 7 * fs;
    auto fx = [&](int64_t c) { return Q::add(Q::curl(Az[c + p1] - Az[c], dy, idy, Ay[c + 1] - Ay[c], dz, idz), S(b0x)); };
    auto fy = [&](int64_t c) { return Q::add(Q::curl(Ax[c + 1] - Ax[c], dz, idz, Az[c + p0] - Az[c], dx, idx), S(b0y)); };
    auto fz = [&](int64_t c) { return Q::add(Q::curl(Ay[c + p0] - Ay[c], dx, idx, Ax[c + p1] - Ax[c], dy, idy), S(b0z)); };
    const S bx = Q::mul(S(0.5), Q::add(fx(o), fx(o + p0)));
    const S by = Q::mul(S(0.5), Q::add(fy(o), fy(o + p1)));
    const S bz = Q::mul(S(0.5), Q::add(fz(o), fz(o + 1)));
    const S r = src[o];
    const S ir = M::inv(r);
    const S u = Q::div(src[fs + o], r, ir), v = Q::div(src[2 * fs + o], r, ir), w = Q::div(src[3 * fs + o], r, ir);
    const S x2 = Q::mul(bx, bx), y2 = Q::mul(by, by), z2 = Q::mul(bz, bz);
    const S xy = Q::add(x2, y2), yz = Q::add(y2, z2), zx = Q::add(z2, x2);
    const S p = rate_pressure(gm1, src[4 * fs + o], r, u, v, w, Q::add(xy, z2));
    const S a2 = Q::quotient(Q::mul(g, p), r, ir);
    const S cx = Q::add(rabs(u), rate_speed<S, 3>(a2, bx, Q::add(xy, z2), r, ir));
    const S cy = Q::add(rabs(v), rate_speed<S, 3>(a2, by, Q::add(yz, x2), r, ir));
    const S cz = Q::add(rabs(w), rate_speed<S, 3>(a2, bz, Q::add(zx, y2), r, ir));
    largest = rmax(largest, Q::ratio_plus(cz, dz, idz, Q::ratio_plus(cx, dx, idx, Q::quotient(cy, dy, idy))));
    smallest = rmin(smallest, r);
  }
}

// The cells of one chunk (kRateChunk cells of patch pi from `chunk_start`) over the NT
// threads of a block, reduced into the chunk's slots: the max / min in the state's type
// (exact: the max of the float rates converts to the max of their double images), converted
// once for the block reduction. 2D:
template <typename S, int NT>
__device__ __forceinline__ void rate_chunk2d(const S* pool, const PatchDesc* patches, int pi,
                                             int chunk_start, double b0x, double b0y, double gamma,
                                             const RateSlots& slots) {
  const PatchDesc P = patches[pi];
  unsigned long long *keys, *level_min;
  if (!rate_slot(P, slots, &keys, &level_min)) return;  // uniform over the block
  S largest = S(0), smallest = S(INFINITY);
  rate_cells2d<S, NT>(pool + P.off, P, unsigned(chunk_start), int(kRateChunk / NT), b0x, b0y, gamma, largest, smallest);
  block_reduce_keys(double(largest), double(smallest), keys, level_min);
}

// 3D:
template <typename S, int NT>
__device__ __forceinline__ void rate_chunk3d(const S* pool, const PatchDesc* patches, int pi,
                                             int chunk_start, double b0x, double b0y, double b0z, double gamma,
                                             const RateSlots& slots) {
  const PatchDesc P = patches[pi];
  unsigned long long *keys, *level_min;
  if (!rate_slot(P, slots, &keys, &level_min)) return;  // uniform over the block
  S largest = S(0), smallest = S(INFINITY);
  rate_cells3d<S, NT>(pool + P.off, P, unsigned(chunk_start), int(kRateChunk / NT), b0x, b0y, b0z, gamma, largest,
                      smallest);
  block_reduce_keys(double(largest), double(smallest), keys, level_min);
}

// dt of instance i: cfl times the smaller of the fast-wave crossing time 1 / rate and the
// explicit diffusion limit 0.5 / (D (dx^-2 + dy^-2 [+ dz^-2])), D = max(eta, (gamma - 1)
// kappa / rho_min). With per-level keys the limit is taken level by level, each level's
// smallest density with that level's spacing, as the reference takes it patch by patch
// (carafe/mhd.py:942-960: patches of one level share the spacing, so the smallest
// density of the level decides); without them, the instance's smallest density with its
// finest spacing.
__device__ __forceinline__ void finalize_dt_one(int i, const unsigned long long* keys, double cfl, double eta,
                                                double kappa, double gamma, const double* inv_dx2_sum,
                                                const unsigned long long* level_keys, const double* inv_dx2_levels,
                                                int nlevels, double* time, const double* end, double* dt,
                                                int advance) {
  const double rate = key_to_double(keys[2 * i]);
  double smallest = 1.0 / rate;
  if (eta > 0.0 || kappa > 0.0) {
    if (level_keys) {
      for (int l = 0; l < nlevels; ++l) {
        const double inv = inv_dx2_levels[i * nlevels + l];
        if (!(inv > 0.0)) continue;  // no patch of the instance on this level
        const double rho_min = key_to_double(level_keys[i * nlevels + l]);
        const double diffusivity = fmax(eta, (gamma - 1.0) * kappa / rho_min);
        if (diffusivity > 0.0) smallest = fmin(smallest, 0.5 / (diffusivity * inv));
      }
    } else {
      const double rho_min = key_to_double(keys[2 * i + 1]);
      const double diffusivity = fmax(eta, (gamma - 1.0) * kappa / rho_min);
      if (diffusivity > 0.0) smallest = fmin(smallest, 0.5 / (diffusivity * inv_dx2_sum[i]));
    }
  }
  double step = cfl * smallest;
  if (end) {
    const double remaining = end[i] - time[i];
    if (!(time[i] < end[i] * (1.0 - 1e-14))) step = 0.0;
    step = fmin(step, fmax(remaining, 0.0));
  }
  dt[i] = step;
  if (advance && time) time[i] += step;
}

}  // namespace wb
