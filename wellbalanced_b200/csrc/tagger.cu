// Learned refinement tagger: stencil features of the 3D state and a small MLP
// (16 -> 64 -> 64 -> 1, ReLU) with bfloat16 weights and float32 accumulation, trained on
// the device. It predicts which cells the plain current tagger (|J| dx > threshold,
// carafe/mhd3d.py:771-801) will flag within the next steps, so a hierarchy can be regridded
// less often. There is no counterpart in the reference; the float64 NumPy restatement in
// oracle/mlp.py is the checker of the forward and backward passes.
//
// Model (the same in every kernel): x^ = bf16(x); z1 = bf16(W1) x^ + b1; h1 = relu(z1);
// z2 = bf16(W2) bf16(h1) + b2; h2 = relu(z2); z = bf16(W3) . h2 + b3. Gradients pass
// through the bf16 roundings unchanged. Parameters live in one float32 buffer:
// W1 [64][16] | b1 [64] | W2 [64][64] | b2 [64] | W3 [64] | b3 [1]  (5313 values).
#include <cuda_bf16.h>

#include <algorithm>

#include "layout.cuh"
#include "numerics.cuh"
#include "stage.cuh"
#include "wb_internal.cuh"

namespace wb {

constexpr int kFeat = 16, kHid = 64;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kHid * kFeat, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid,
              kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid, kParams = kOffB3 + 1;
static_assert(kParams == 5313, "parameter layout");

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// ---- features ------------------------------------------------------------------------------------
// (log rho, log p, |B|) of haloed cell (i, j, k) of a 3D patch (cell B = mean of its face fields
// from the curl of the edge potential, as the stage kernels form it).
template <typename S>
__device__ __forceinline__ void cell_quantities(const S* src, const PatchDesc& P, int i, int j, int k,
                                                const double* b0, double gamma, float (&q)[3]) {
  using M = Math<S>;
  const int64_t p0 = P.pitch0, p1 = P.pitch1, fs = P.fstride;
  const int64_t o = int64_t(i) * p0 + int64_t(j) * p1 + k;
  const S* Ax = src + 5 * fs;
  const S* Ay = src + 6 * fs;
  const S* Az = src + 7 * fs;
  const S dx = S(P.dx[0]), dy = S(P.dx[1]), dz = S(P.dx[2]);
  const S idx = M::inv(dx), idy = M::inv(dy), idz = M::inv(dz);
  auto fx = [&](int64_t c) { return M::div(Az[c + p1] - Az[c], dy, idy) - M::div(Ay[c + 1] - Ay[c], dz, idz) + S(b0[0]); };
  auto fy = [&](int64_t c) { return M::div(Ax[c + 1] - Ax[c], dz, idz) - M::div(Az[c + p0] - Az[c], dx, idx) + S(b0[1]); };
  auto fz = [&](int64_t c) { return M::div(Ay[c + p0] - Ay[c], dx, idx) - M::div(Ax[c + p1] - Ax[c], dy, idy) + S(b0[2]); };
  const S bx = S(0.5) * (fx(o) + fx(o + p0));
  const S by = S(0.5) * (fy(o) + fy(o + p1));
  const S bz = S(0.5) * (fz(o) + fz(o + 1));
  const S r = src[o];
  const S m0 = src[fs + o], m1 = src[2 * fs + o], m2 = src[3 * fs + o], e = src[4 * fs + o];
  const S ir = M::inv(r);
  const S p = recover_pressure<S>(r, m0, m1, m2, e, bx, by, bz, m0 * ir, m1 * ir, m2 * ir, gamma);
  q[0] = logf(fmaxf(float(r), 1e-30f));
  q[1] = logf(fmaxf(float(p), 1e-30f));
  q[2] = sqrtf(float(bx * bx + by * by + bz * bz));
}

// Features of a cell from its 3 x 3 x 3 neighbourhood, for each of (log rho, log p, |B|):
// the value, the three central differences (half the difference of the two neighbours
// along an axis) and the largest deviation over the 26 neighbours; feature 15 is zero.
// Output row t of a patch's block is its cell (i, j, k) in (i, j, k) order, normalised
// as (f - mean) * inv_std. Work list of the rate kernels: up to 2048 cells per chunk.
//
// The quantities of a cell (two logarithms, a root, the float64 pressure, 17 loads) are what a
// cell costs: forming those of all 27 neighbours by every thread took 27 of them a row. A
// block takes 512 consecutive cells, forms each quantity of their neighbourhood once in
// shared memory (about 4 a row) and then the stencils. The neighbourhood is the box of
// planes, rows and whole z-lines around the cells where that fits the 72 KB (three blocks of
// 512 threads an SM): z up to 510 cells inside one plane, patches of up to 24 x 24 across
// planes; other cells go row by row, three lines of three rows each.
// B200, 491,000 cells in 203 patches: 195 -> 50 us.
constexpr int kTagCells = 512;
constexpr int kTagRegion = 6144;  // cells of the neighbourhood held at once
constexpr size_t kTagSmem = 3 * kTagRegion * sizeof(float);

template <typename S>
__global__ void __launch_bounds__(kTagCells) tag_features3d_kernel(const S* __restrict__ pool, const PatchDesc* patches,
                                                                   const int* chunk_patch, const int* chunk_start,
                                                                   const int64_t* row_start, double b0x, double b0y,
                                                                   double b0z, double gamma, const float* mean,
                                                                   const float* inv_std, float* __restrict__ out) {
  extern __shared__ float q[];  // [3][kTagRegion]
  constexpr int kParts = 2048 / kTagCells;
  const int chunk = int(blockIdx.x) / kParts, part = int(blockIdx.x) % kParts;
  const int pi = chunk_patch[chunk];
  const PatchDesc P = patches[pi];
  const int nx = P.n[0], ny = P.n[1], nz = P.n[2];
  const S* src = pool + P.off;
  const double b0[3] = {b0x, b0y, b0z};
  const unsigned total = unsigned(nx) * unsigned(ny) * unsigned(nz);
  const unsigned begin = unsigned(chunk_start[chunk]) + unsigned(part) * kTagCells;
  if (begin >= total) return;
  const unsigned end = min(begin + unsigned(kTagCells), total);
  for (unsigned first = begin; first < end;) {
    // the segment [first, last) and its box of neighbours: planes i0 - 1 .. i1 + 1, rows
    // j0 - 1 .. j1 + 1, cells k0 - 1 .. k1 + 1 of the interior indices
    unsigned last = end;
    const unsigned line0 = first / unsigned(nz);
    unsigned line1 = (last - 1) / unsigned(nz);
    int i0 = int(line0 / unsigned(ny)), j0 = int(line0 - unsigned(i0) * unsigned(ny)), k0 = 0;
    int i1 = int(line1 / unsigned(ny)), j1 = int(line1 - unsigned(i1) * unsigned(ny)), k1 = nz - 1;
    if (i1 > i0) j1 = ny - 1;
    const int jb = i1 > i0 ? 0 : j0;
    int64_t cells = int64_t(i1 - i0 + 3) * (j1 - jb + 3) * (int64_t(nz) + 2);
    if (cells <= kTagRegion) {
      j0 = jb;
    } else {  // one row at a time, its part of the line only
      last = min(end, (line0 + 1) * unsigned(nz));
      i1 = i0;
      j1 = j0;
      k0 = int(first - line0 * unsigned(nz));
      k1 = int(last - 1 - line0 * unsigned(nz));
      cells = int64_t(3) * 3 * (k1 - k0 + 3);  // at most 9 x 514
    }
    const int width = k1 - k0 + 3, rows = j1 - j0 + 3;
    for (int t = threadIdx.x; t < int(cells); t += kTagCells) {
      const int line = t / width, k = t - line * width;
      const int plane = line / rows, j = line - plane * rows;
      float v[3];
      cell_quantities<S>(src, P, i0 - 1 + plane + kHalo, j0 - 1 + j + kHalo, k0 - 1 + k + kHalo, b0, gamma, v);
      q[t] = v[0];
      q[kTagRegion + t] = v[1];
      q[2 * kTagRegion + t] = v[2];
    }
    __syncthreads();
    const unsigned t = first + threadIdx.x;
    if (t < last) {
      const unsigned line = t / unsigned(nz);
      const int i = int(line / unsigned(ny));
      const int j = int(line - unsigned(i) * unsigned(ny)), k = int(t - line * unsigned(nz));
      const int at = ((i - i0 + 1) * rows + (j - j0 + 1)) * width + (k - k0 + 1);
      const int sj = width, si = rows * width;
      float f[kFeat];
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        const float* c = q + v * kTagRegion + at;
        const float c0 = c[0];
        float dev = 0.0f;
#pragma unroll
        for (int a = -1; a <= 1; ++a)
#pragma unroll
          for (int b = -1; b <= 1; ++b)
#pragma unroll
            for (int d = -1; d <= 1; ++d) dev = fmaxf(dev, fabsf(c[a * si + b * sj + d] - c0));
        f[v] = c0;
        f[3 + 3 * v + 0] = 0.5f * (c[si] - c[-si]);
        f[3 + 3 * v + 1] = 0.5f * (c[sj] - c[-sj]);
        f[3 + 3 * v + 2] = 0.5f * (c[1] - c[-1]);
        f[12 + v] = dev;
      }
      f[15] = 0.0f;
      float* row = out + (row_start[pi] + int64_t(t)) * kFeat;
#pragma unroll
      for (int c = 0; c < kFeat; ++c) f[c] = (f[c] - mean[c]) * inv_std[c];
      if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {  // uniform: rows are 64 bytes
#pragma unroll
        for (int c = 0; c < kFeat; c += 4)
          *reinterpret_cast<float4*>(row + c) = make_float4(f[c], f[c + 1], f[c + 2], f[c + 3]);
      } else {
#pragma unroll
        for (int c = 0; c < kFeat; ++c) row[c] = f[c];
      }
    }
    __syncthreads();
    first = last;
  }
}

// ---- forward on the tensor cores --------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// D = A (16 x 16, row) * B (16 x 8, col) + D; bf16 inputs, float32 accumulation.
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Padded row pitches (in bf16) of the weights in shared memory: rows 16 B apart modulo 128 B,
// so the 8 rows a fragment load touches fall in different banks.
constexpr int kPitch1 = kFeat + 8, kPitch2 = kHid + 8;

// Each warp takes 16 rows at a time: layer 1 as 8 mma (one per 8 outputs), layer 2 as
// 32 mma with the layer-1 accumulators re-packed in registers as its A fragments
// (the accumulator layout of m16n8 matches the A layout of the next k-tile), layer 3 as
// a dot product reduced over the four threads that hold a row.
__global__ void __launch_bounds__(256) mlp_forward_kernel(const float* __restrict__ X, int64_t n,
                                                          const float* __restrict__ params,
                                                          float* __restrict__ logits) {
  __shared__ __align__(16) __nv_bfloat16 sW1[kHid * kPitch1];
  __shared__ __align__(16) __nv_bfloat16 sW2[kHid * kPitch2];
  __shared__ float sB1[kHid], sB2[kHid], sW3[kHid];
  for (int t = threadIdx.x; t < kHid * kFeat; t += blockDim.x)
    sW1[(t / kFeat) * kPitch1 + t % kFeat] = __float2bfloat16_rn(params[kOffW1 + t]);
  for (int t = threadIdx.x; t < kHid * kHid; t += blockDim.x)
    sW2[(t / kHid) * kPitch2 + t % kHid] = __float2bfloat16_rn(params[kOffW2 + t]);
  for (int t = threadIdx.x; t < kHid; t += blockDim.x) {
    sB1[t] = params[kOffB1 + t];
    sB2[t] = params[kOffB2 + t];
    sW3[t] = bf16r(params[kOffW3 + t]);
  }
  __syncthreads();
  const float b3 = params[kOffB3];
  const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t tile = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); tile * 16 < n; tile += warps) {
    const int64_t r0 = tile * 16 + g, r1 = r0 + 8;
    auto x = [&](int64_t r, int c) { return r < n ? X[r * kFeat + c] : 0.0f; };
    uint32_t a[4];
    a[0] = pack_bf16(x(r0, 2 * tg), x(r0, 2 * tg + 1));
    a[1] = pack_bf16(x(r1, 2 * tg), x(r1, 2 * tg + 1));
    a[2] = pack_bf16(x(r0, 2 * tg + 8), x(r0, 2 * tg + 9));
    a[3] = pack_bf16(x(r1, 2 * tg + 8), x(r1, 2 * tg + 9));
    float h1[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const int col = nt * 8 + 2 * tg;
      h1[nt][0] = h1[nt][2] = sB1[col];
      h1[nt][1] = h1[nt][3] = sB1[col + 1];
      const __nv_bfloat16* w = sW1 + (nt * 8 + g) * kPitch1 + 2 * tg;
      mma_bf16(h1[nt], a, *reinterpret_cast<const uint32_t*>(w), *reinterpret_cast<const uint32_t*>(w + 8));
#pragma unroll
      for (int e = 0; e < 4; ++e) h1[nt][e] = fmaxf(h1[nt][e], 0.0f);
    }
    float h2[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const int col = nt * 8 + 2 * tg;
      h2[nt][0] = h2[nt][2] = sB2[col];
      h2[nt][1] = h2[nt][3] = sB2[col + 1];
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t a2[4];
      a2[0] = pack_bf16(h1[2 * kk][0], h1[2 * kk][1]);
      a2[1] = pack_bf16(h1[2 * kk][2], h1[2 * kk][3]);
      a2[2] = pack_bf16(h1[2 * kk + 1][0], h1[2 * kk + 1][1]);
      a2[3] = pack_bf16(h1[2 * kk + 1][2], h1[2 * kk + 1][3]);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const __nv_bfloat16* w = sW2 + (nt * 8 + g) * kPitch2 + kk * 16 + 2 * tg;
        mma_bf16(h2[nt], a2, *reinterpret_cast<const uint32_t*>(w), *reinterpret_cast<const uint32_t*>(w + 8));
      }
    }
    float z0 = 0.0f, z1 = 0.0f;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const int col = nt * 8 + 2 * tg;
      z0 += fmaxf(h2[nt][0], 0.0f) * sW3[col] + fmaxf(h2[nt][1], 0.0f) * sW3[col + 1];
      z1 += fmaxf(h2[nt][2], 0.0f) * sW3[col] + fmaxf(h2[nt][3], 0.0f) * sW3[col + 1];
    }
    z0 += __shfl_xor_sync(0xffffffffu, z0, 1);
    z0 += __shfl_xor_sync(0xffffffffu, z0, 2);
    z1 += __shfl_xor_sync(0xffffffffu, z1, 1);
    z1 += __shfl_xor_sync(0xffffffffu, z1, 2);
    if (tg == 0) {
      if (r0 < n) logits[r0] = z0 + b3;
      if (r1 < n) logits[r1] = z1 + b3;
    }
  }
}

// ---- backward on the CUDA cores -----------------------------------------------------------------------
// 256 threads and 64 samples per round: five small matrix products (Z1, Z2 forward, D1 back,
// the gradients of W2 and W1), each 64 x 64 (or x 16), as 4 x 4 tiles of a thread over
// operands stored in shared memory with the summed index outermost: two 16-byte loads feed
// 16 multiply-adds. Deltas and sums stay float32 (tensor cores would take them in 16 bits);
// a sum runs over its index in order. dL/dz = w (sigmoid(z) - y) of the weighted binary
// cross-entropy (w = pos_weight for y = 1). Weight gradients stay in registers over a
// block's rounds; each block adds its sums to `grads` (float32, parameter layout) once, four
// values per reduction, `loss` (float64) gets the summed loss. One block an SM, so that 148
// blocks' sums meet in L2 instead of one per round. B200, 16384 samples: 103 us with one
// multiply-add per two 4-byte shared-memory loads, 28 us now (3.6 us a round of
// multiply-adds at full rate, two rounds).
constexpr int kRound = 64;
constexpr int kPitch = kHid + 4;   // row pitch of the 64 x 64 operands: 16-byte rows, 4 banks apart
constexpr int kPitchX = kFeat + 4;
constexpr int kSquare = kHid * kPitch;
constexpr size_t kBackwardSmem = sizeof(float) * (kFeat * kHid + 7 * kSquare + 3 * kHid + kRound * kPitchX + kFeat * kPitch);

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
}

// acc[a][b] += sum over `count` k of A[k][4 row + a] B[k][4 col + b], k in order.
__device__ __forceinline__ void tile_product(const float* A, int pitch_a, const float* B, int pitch_b, int count,
                                             float (&acc)[4][4]) {
#pragma unroll 4
  for (int k = 0; k < count; ++k) {
    float x[4], w[4];
    load4(A + k * pitch_a, x);
    load4(B + k * pitch_b, w);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(w[b], x[a], acc[a][b]);
  }
}

// A 4 x 4 tile into row-major rows and, transposed, into column-major ones.
__device__ __forceinline__ void store_tile(float* rows, const float (&v)[4][4]) {
#pragma unroll
  for (int a = 0; a < 4; ++a) *reinterpret_cast<float4*>(rows + a * kPitch) = make_float4(v[a][0], v[a][1], v[a][2], v[a][3]);
}
__device__ __forceinline__ void store_transposed(float* cols, const float (&v)[4][4]) {
#pragma unroll
  for (int b = 0; b < 4; ++b) *reinterpret_cast<float4*>(cols + b * kPitch) = make_float4(v[0][b], v[1][b], v[2][b], v[3][b]);
}

// Adds four consecutive values to global memory: one reduction where they are 16-byte aligned.
__device__ __forceinline__ void add4(float* p, const float (&v)[4]) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                 : "memory");
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) atomicAdd(p + e, v[e]);
  }
}

__global__ void __launch_bounds__(256) mlp_backward_kernel(const float* __restrict__ X, const float* __restrict__ y,
                                                           int64_t n, const float* __restrict__ params,
                                                           float pos_weight, float* __restrict__ grads,
                                                           double* __restrict__ loss) {
  extern __shared__ __align__(16) float smem[];
  float* sW1T = smem;                    // [16][64] bf16-rounded W1, [in][out]
  float* sW2 = sW1T + kFeat * kHid;      // [out][in]
  float* sW2T = sW2 + kSquare;           // [in][out]
  float* sH1 = sW2T + kSquare;           // [sample][unit] bf16(h1)
  float* sH1T = sH1 + kSquare;           // [unit][sample]
  float* sD2 = sH1T + kSquare;           // [sample][unit]
  float* sD2T = sD2 + kSquare;           // [unit][sample]
  float* sD1 = sD2T + kSquare;           // [sample][unit]
  float* sB1 = sD1 + kSquare;
  float* sB2 = sB1 + kHid;
  float* sW3 = sB2 + kHid;
  float* sX = sW3 + kHid;                // [sample][feature]
  float* sXT = sX + kRound * kPitchX;    // [feature][sample]
  __shared__ double sLoss[8];
  const int tid = threadIdx.x;
  for (int t = tid; t < kHid * kFeat; t += 256) sW1T[(t % kFeat) * kHid + t / kFeat] = bf16r(params[kOffW1 + t]);
  for (int t = tid; t < kHid * kHid; t += 256) {
    const float w = bf16r(params[kOffW2 + t]);
    sW2[(t / kHid) * kPitch + t % kHid] = w;
    sW2T[(t % kHid) * kPitch + t / kHid] = w;
  }
  if (tid < kHid) {
    sB1[tid] = params[kOffB1 + tid];
    sB2[tid] = params[kOffB2 + tid];
    sW3[tid] = bf16r(params[kOffW3 + tid]);
  }
  const float b3 = params[kOffB3];
  // tiles: samples (or units) 4 row .., units 4 col ..; of W1's gradient: a quarter of the
  // samples, units 4 wj .., features 4 wc ..
  const int row = tid >> 4, col = tid & 15;
  const int quarter = tid >> 6, wj = (tid & 63) >> 2, wc = tid & 3;
  float gw2[4][4] = {}, gw1[4][4] = {}, gw3[4] = {}, gb1[4] = {}, gb2[4] = {}, gb3 = 0.0f;
  double my_loss = 0.0;
  for (int64_t base = int64_t(blockIdx.x) * kRound; base < n; base += int64_t(gridDim.x) * kRound) {
    {
      const int s = tid >> 2, c0 = (tid & 3) * 4;
      const int64_t r = base + s;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float x = r < n ? bf16r(X[r * kFeat + c0 + c]) : 0.0f;
        sX[s * kPitchX + c0 + c] = x;
        sXT[(c0 + c) * kPitch + s] = x;
      }
    }
    __syncthreads();
    float bias[4], w3[4], acc[4][4];
    load4(sB1 + 4 * col, bias);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = bias[b];
    tile_product(sXT + 4 * row, kPitch, sW1T + 4 * col, kHid, kFeat, acc);
    unsigned active1 = 0;  // units with z1 > 0
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        active1 |= acc[a][b] > 0.0f ? 1u << (4 * a + b) : 0u;
        acc[a][b] = bf16r(fmaxf(acc[a][b], 0.0f));
      }
    store_tile(sH1 + 4 * row * kPitch + 4 * col, acc);
    store_transposed(sH1T + 4 * col * kPitch + 4 * row, acc);
    __syncthreads();
    load4(sB2 + 4 * col, bias);
    load4(sW3 + 4 * col, w3);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = bias[b];
    tile_product(sH1T + 4 * row, kPitch, sW2T + 4 * col, kPitch, kHid, acc);
    // output, loss and deltas of the tile's samples
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      float z = 0.0f;
#pragma unroll
      for (int b = 0; b < 4; ++b) z = fmaf(fmaxf(acc[a][b], 0.0f), w3[b], z);
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
      z += b3;
      const int64_t r = base + 4 * row + a;
      const bool live = r < n;
      const float target = live ? y[r] : 0.0f;
      const float w = target > 0.5f ? pos_weight : 1.0f;
      const float prob = 1.0f / (1.0f + __expf(-z));
      const float d3 = live ? w * (prob - target) : 0.0f;
      if (col == 0) {
        gb3 += d3;
        // softplus(z) - y z, evaluated without overflow
        const float sp = fmaxf(z, 0.0f) + log1pf(__expf(-fabsf(z)));
        my_loss += live ? double(w) * double(sp - target * z) : 0.0;
      }
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        gw3[b] = fmaf(d3, fmaxf(acc[a][b], 0.0f), gw3[b]);
        acc[a][b] = acc[a][b] > 0.0f ? d3 * w3[b] : 0.0f;
        gb2[b] += acc[a][b];
      }
    }
    store_tile(sD2 + 4 * row * kPitch + 4 * col, acc);
    store_transposed(sD2T + 4 * col * kPitch + 4 * row, acc);
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = 0.0f;
    tile_product(sD2T + 4 * row, kPitch, sW2 + 4 * col, kPitch, kHid, acc);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        acc[a][b] = active1 >> (4 * a + b) & 1u ? acc[a][b] : 0.0f;
        gb1[b] += acc[a][b];
      }
    store_tile(sD1 + 4 * row * kPitch + 4 * col, acc);
    tile_product(sD2 + 4 * row, kPitch, sH1 + 4 * col, kPitch, kRound, gw2);
    __syncthreads();
    tile_product(sD1 + quarter * 16 * kPitch + 4 * wj, kPitch, sX + quarter * 16 * kPitchX + 4 * wc, kPitchX, 16, gw1);
    __syncthreads();
  }
  // the block's sums: W2's tiles as they are; W1's over the quarters, the unit sums over the
  // 16 rows of tiles, through shared memory
#pragma unroll
  for (int a = 0; a < 4; ++a) add4(grads + kOffW2 + (4 * row + a) * kHid + 4 * col, gw2[a]);
  float* sW1G = sH1;           // [4][64][16]
  float* sSums = sD2;          // [3][16][64]
#pragma unroll
  for (int a = 0; a < 4; ++a)
    *reinterpret_cast<float4*>(sW1G + quarter * kHid * kFeat + (4 * wj + a) * kFeat + 4 * wc) =
        make_float4(gw1[a][0], gw1[a][1], gw1[a][2], gw1[a][3]);
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    sSums[row * kHid + 4 * col + b] = gw3[b];
    sSums[16 * kHid + row * kHid + 4 * col + b] = gb1[b];
    sSums[32 * kHid + row * kHid + 4 * col + b] = gb2[b];
  }
  // (the gb3 and loss of a row of tiles sit in its col 0 thread)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
    my_loss += __shfl_xor_sync(0xffffffffu, my_loss, o);
  }
  if ((tid & 31) == 0) {
    sLoss[tid >> 5] = my_loss;
    atomicAdd(&grads[kOffB3], gb3);
  }
  __syncthreads();
  {
    float v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float* g = sW1G + 4 * tid + e;
      v[e] = ((g[0] + g[kHid * kFeat]) + g[2 * kHid * kFeat]) + g[3 * kHid * kFeat];
    }
    add4(grads + kOffW1 + 4 * tid, v);
  }
  if (tid < 3 * kHid) {
    const int which = tid / kHid, unit = tid % kHid;
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < 16; ++k) sum += sSums[(which * 16 + k) * kHid + unit];
    atomicAdd(&grads[(which == 0 ? kOffW3 : which == 1 ? kOffB1 : kOffB2) + unit], sum);
  }
  if (tid == 0) {
    double total = 0.0;
    for (int w = 0; w < 8; ++w) total += sLoss[w];
    atomicAdd(loss, total);
  }
}

// Adam on the float32 parameters with gradients scaled by `scale` (1 / batch size); the
// gradients are cleared for the next accumulation.
__global__ void mlp_adam_kernel(float* params, float* grads, float* m, float* v, int count, float lr, float beta1,
                                float beta2, float eps, float bias1, float bias2, float scale) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const float g = grads[t] * scale;
  const float mt = beta1 * m[t] + (1.0f - beta1) * g;
  const float vt = beta2 * v[t] + (1.0f - beta2) * g * g;
  m[t] = mt;
  v[t] = vt;
  params[t] -= lr * (mt / bias1) / (sqrtf(vt / bias2) + eps);
  grads[t] = 0.0f;
}

}  // namespace wb

// ---- C ABI ---------------------------------------------------------------------------------------
using namespace wb;

extern "C" int wb_tag_features(int precision, const void* pool, const void* patches, const int* chunk_patch,
                               const int* chunk_start, int nchunks, const int64_t* row_start, double b0x, double b0y,
                               double b0z, double gamma, const float* mean, const float* inv_std, float* out,
                               void* stream) {
  set_error("");
  if (!pool || !patches || !row_start || !mean || !inv_std || !out || (nchunks > 0 && (!chunk_patch || !chunk_start))) {
    set_error("tag_features: null pointer");
    return kBadArgument;
  }
  if (nchunks <= 0) return kOk;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int grid = nchunks * (2048 / kTagCells);
  if (precision == 32) {
    cudaFuncSetAttribute(tag_features3d_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTagSmem));
    tag_features3d_kernel<float><<<grid, kTagCells, kTagSmem, s>>>(
        static_cast<const float*>(pool), static_cast<const PatchDesc*>(patches), chunk_patch, chunk_start, row_start,
        b0x, b0y, b0z, gamma, mean, inv_std, out);
  } else if (precision == 64 || precision == kMath32State64) {  // a float64 state
    cudaFuncSetAttribute(tag_features3d_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTagSmem));
    tag_features3d_kernel<double><<<grid, kTagCells, kTagSmem, s>>>(
        static_cast<const double*>(pool), static_cast<const PatchDesc*>(patches), chunk_patch, chunk_start, row_start,
        b0x, b0y, b0z, gamma, mean, inv_std, out);
  }
  else {
    set_error("tag_features: precision is 32, 64 or %d, not %d", kMath32State64, precision);
    return kBadArgument;
  }
  return check_launch("tag_features");
}

extern "C" int wb_mlp_forward(const float* features, int64_t n, const float* params, float* logits, void* stream) {
  set_error("");
  if (!features || !params || !logits || n < 0) {
    set_error("mlp_forward: null pointer or negative row count");
    return kBadArgument;
  }
  if (n == 0) return kOk;
  const int64_t tiles = (n + 15) / 16;
  const int blocks = int(std::min<int64_t>((tiles + 7) / 8, 148 * 8));
  mlp_forward_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(features, n, params, logits);
  return check_launch("mlp_forward");
}

extern "C" int wb_mlp_backward(const float* features, const float* targets, int64_t n, const float* params,
                               float pos_weight, float* grads, double* loss, void* stream) {
  set_error("");
  if (!features || !targets || !params || !grads || !loss || n < 0) {
    set_error("mlp_backward: null pointer or negative row count");
    return kBadArgument;
  }
  if (n == 0) return kOk;
  const int blocks = int(std::min<int64_t>((n + kRound - 1) / kRound, 148));
  cudaFuncSetAttribute(mlp_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBackwardSmem));
  mlp_backward_kernel<<<blocks, 256, kBackwardSmem, static_cast<cudaStream_t>(stream)>>>(
      features, targets, n, params, pos_weight, grads, loss);
  return check_launch("mlp_backward");
}

extern "C" int wb_mlp_adam(float* params, float* grads, float* m, float* v, int count, float lr, float beta1,
                           float beta2, float eps, int step, float scale, void* stream) {
  set_error("");
  if (!params || !grads || !m || !v || count != kParams || step < 1) {
    set_error("mlp_adam: null pointer, parameter count other than %d, or step < 1", kParams);
    return kBadArgument;
  }
  const float bias1 = 1.0f - powf(beta1, float(step)), bias2 = 1.0f - powf(beta2, float(step));
  mlp_adam_kernel<<<(count + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      params, grads, m, v, count, lr, beta1, beta2, eps, bias1, bias2, scale);
  return check_launch("mlp_adam");
}
