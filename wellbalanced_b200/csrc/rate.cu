// Stable time step on device: the fast-wave rate of every cell reduced per instance
// (carafe/kernels/mhd_rate/mhd_rate_pyccel.py:30-83 in 2D, carafe/mhd3d.py:674-724 in
// 3D), then dt = cfl / max rate with the diffusion limit (carafe/mhd.py:930-963).
// Works on the patch pool; no host synchronisation, so a step can be captured in a graph.
// The per-chunk and per-instance bodies are in ratecell.cuh.
#include "layout.cuh"
#include "numerics.cuh"
#include "ratecell.cuh"
#include "stage.cuh"
#include "wb_internal.cuh"

namespace wb {

__global__ void init_keys_kernel(unsigned long long* keys) {
  keys[0] = double_to_key(0.0);
  keys[1] = rate_min_identity();
}

// Reduction identities of n instances' (max rate, min density) keys and, when
// level_keys is given, of their per-level density minima (n x nlevels keys).
__global__ void init_keys_n_kernel(unsigned long long* keys, int n, unsigned long long* level_keys, int nlevels) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    keys[2 * i] = double_to_key(0.0);
    keys[2 * i + 1] = rate_min_identity();
  }
  if (level_keys && i < n * nlevels) level_keys[i] = rate_min_identity();
}

constexpr int kRateThreads = 256;  // threads of a rate block (8 rounds: 2048 cells)

// One block per (patch, chunk of cells).
template <typename S>
__global__ void __launch_bounds__(kRateThreads) rate2d_kernel(const S* __restrict__ pool, const PatchDesc* patches,
                                                    int npatches, const int* chunk_patch,
                                                    const int* chunk_start, double b0x, double b0y,
                                                    double gamma, const RateSlots slots) {
  rate_chunk2d<S, kRateThreads>(pool, patches, chunk_patch[blockIdx.x], chunk_start[blockIdx.x], b0x, b0y, gamma,
                                slots);
}

template <typename S>
__global__ void __launch_bounds__(kRateThreads) rate3d_kernel(const S* __restrict__ pool, const PatchDesc* patches,
                                                    int npatches, const int* chunk_patch,
                                                    const int* chunk_start, double b0x, double b0y,
                                                    double b0z, double gamma, const RateSlots slots) {
  rate_chunk3d<S, kRateThreads>(pool, patches, chunk_patch[blockIdx.x], chunk_start[blockIdx.x], b0x, b0y, b0z,
                                gamma, slots);
}

// The work list of the rate kernels is derived from the patch table on the host and
// kept by the caller (chunks of 2048 cells).
template <typename S>
int launch_rate_chunks(const S* state, const PatchDesc* patches, int npatches, int ndim, const int* chunk_patch,
                       const int* chunk_start, int nchunks, const double* b0, double gamma,
                       unsigned long long* keys, int ninstances, cudaStream_t stream,
                       unsigned long long* level_keys, int nlevels, unsigned* error) {
  const int slots_n = level_keys ? max(ninstances, ninstances * nlevels) : ninstances;
  init_keys_n_kernel<<<(slots_n + 255) / 256, 256, 0, stream>>>(keys, ninstances, level_keys, nlevels);
  const RateSlots slots{keys, ninstances, level_keys, nlevels, error};
  if (nchunks > 0) {
    if (ndim == 2)
      rate2d_kernel<S><<<nchunks, kRateThreads, 0, stream>>>(state, patches, npatches, chunk_patch, chunk_start, b0[0], b0[1],
                                                    gamma, slots);
    else
      rate3d_kernel<S><<<nchunks, kRateThreads, 0, stream>>>(state, patches, npatches, chunk_patch, chunk_start, b0[0], b0[1],
                                                    b0[2], gamma, slots);
  }
  return check_launch("rate");
}

template int launch_rate_chunks<float>(const float*, const PatchDesc*, int, int, const int*, const int*, int,
                                       const double*, double, unsigned long long*, int, cudaStream_t,
                                       unsigned long long*, int, unsigned*);
template int launch_rate_chunks<double>(const double*, const PatchDesc*, int, int, const int*, const int*, int,
                                        const double*, double, unsigned long long*, int, cudaStream_t,
                                        unsigned long long*, int, unsigned*);

__global__ void finalize_dt_kernel(const unsigned long long* keys, int n, double cfl, double eta, double kappa,
                                   double gamma, const double* inv_dx2_sum, const unsigned long long* level_keys,
                                   const double* inv_dx2_levels, int nlevels, double* time, const double* end,
                                   double* dt, int advance) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    finalize_dt_one(i, keys, cfl, eta, kappa, gamma, inv_dx2_sum, level_keys, inv_dx2_levels, nlevels, time, end, dt,
                    advance);
}

int launch_finalize_dt(const unsigned long long* keys, int ninstances, double cfl, double eta, double kappa,
                       double gamma, const double* inv_dx2_sum, double* time, const double* end, double* dt,
                       int advance_time, cudaStream_t stream, const unsigned long long* level_keys,
                       const double* inv_dx2_levels, int nlevels) {
  if (ninstances > 0)
    finalize_dt_kernel<<<(ninstances + 255) / 256, 256, 0, stream>>>(keys, ninstances, cfl, eta, kappa, gamma,
                                                                     inv_dx2_sum, level_keys, inv_dx2_levels,
                                                                     nlevels, time, end, dt, advance_time);
  return check_launch("finalize_dt");
}

// The stable step in one launch: `parts` blocks share each 2048-cell chunk of the work list;
// a block reduces its cells, takes the maximum and minimum to the scratch keys (an atomic only
// where it would change the key), and the last block to finish turns the keys into every
// instance's dt, hands them on in `keys` / `level_keys` and puts the scratch back to the
// identities for the next launch. Three launches (keys, rate, dt) and 8 serial rounds a block
// before; small grids, whose few chunks left most SMs idle, take 8 blocks a chunk. B200, the
// three launches and this one: a 32^2 float64 grid 9.7 and 6.0 us, 256^2 14.2 and 7.2, a 256^3
// float32 box 194 and 162, 512 2D float32 instances 95 and 98 (bound by the reads of the state
// and the latency of the chain behind them; the batch's blocks by their look-ups).
struct StableDt {
  double cfl, eta, kappa, gamma;
  const double *inv_dx2_sum, *inv_dx2_levels;
  double* time;
  const double* end;
  double* dt;
  int advance;
  unsigned long long *keys, *level_keys;  // the results (level_keys nullable)
};

// (float32: 32 registers, 64 warps an SM, as the rate kernel alone)
template <typename S, int NDIM>
__global__ void __launch_bounds__(kRateThreads, sizeof(S) == 4 ? 8 : 4)
    stable_dt_kernel(const S* pool, const PatchDesc* patches, const int* chunk_patch, const int* chunk_start,
                     int nchunks, int parts, double b0x, double b0y, double b0z, const RateSlots scratch,
                     unsigned* ticket, const StableDt a) {
  after_previous();
  __shared__ double s_largest[kRateThreads / 32], s_smallest[kRateThreads / 32];
  __shared__ bool s_last;
  const int chunk = int(blockIdx.x) / parts, part = int(blockIdx.x) - chunk * parts;
  if (chunk < nchunks) {
    const PatchDesc P = patches[chunk_patch[chunk]];
    unsigned long long *keys, *level_min;
    if (rate_slot(P, scratch, &keys, &level_min)) {  // uniform over the block
      const int rounds = int(kRateChunk / kRateThreads) / parts;
      const unsigned begin = unsigned(chunk_start[chunk]) + unsigned(part * rounds * kRateThreads);
      S largest = S(0), smallest = S(INFINITY);
      if (NDIM == 2)
        rate_cells2d<S, kRateThreads>(pool + P.off, P, begin, rounds, b0x, b0y, a.gamma, largest, smallest);
      else
        rate_cells3d<S, kRateThreads>(pool + P.off, P, begin, rounds, b0x, b0y, b0z, a.gamma, largest, smallest);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        largest = rmax(largest, __shfl_xor_sync(0xffffffffu, largest, o));
        smallest = rmin(smallest, __shfl_xor_sync(0xffffffffu, smallest, o));
      }
      if ((threadIdx.x & 31) == 0) {
        s_largest[threadIdx.x >> 5] = double(largest);
        s_smallest[threadIdx.x >> 5] = double(smallest);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        double top = s_largest[0], low = s_smallest[0];
#pragma unroll
        for (int w = 1; w < kRateThreads / 32; ++w) {
          top = fmax(top, s_largest[w]);
          low = fmin(low, s_smallest[w]);
        }
        const unsigned long long kt = double_to_key(top), kl = double_to_key(low);
        if (kt > *static_cast<volatile unsigned long long*>(keys)) atomicMax(keys, kt);
        if (kl < *static_cast<volatile unsigned long long*>(keys + 1)) atomicMin(keys + 1, kl);
        if (level_min && kl < *static_cast<volatile unsigned long long*>(level_min)) atomicMin(level_min, kl);
      }
    }
  }
  if (threadIdx.x == 0) {
    __threadfence();  // the block's keys before its ticket
    // counts to the grid's size and wraps to zero by itself: two launches that overlap spoil
    // their own dt, and the scratch is whole again when both have finished
    s_last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();  // the other blocks' keys after their tickets
  const int n = scratch.ninstances, nlevels = scratch.nlevels;
  for (int i = threadIdx.x; i < n; i += kRateThreads) {
    a.keys[2 * i] = __ldcg(scratch.keys + 2 * i);
    a.keys[2 * i + 1] = __ldcg(scratch.keys + 2 * i + 1);
    scratch.keys[2 * i] = double_to_key(0.0);
    scratch.keys[2 * i + 1] = rate_min_identity();
    if (scratch.level_keys)
      for (int l = 0; l < nlevels; ++l) {
        a.level_keys[i * nlevels + l] = __ldcg(scratch.level_keys + i * nlevels + l);
        scratch.level_keys[i * nlevels + l] = rate_min_identity();
      }
    finalize_dt_one(i, a.keys, a.cfl, a.eta, a.kappa, a.gamma, a.inv_dx2_sum, a.level_keys, a.inv_dx2_levels, nlevels,
                    a.time, a.end, a.dt, a.advance);
  }
}

// Instances up to which the last block makes every dt. More take the rate and dt launches: one
// block walks them 256 at a time, and thousands of small blocks queue at the ticket. B200,
// three launches and one, float32 (float64): 256 instances of 64^2 12.2 and 12.0 us (21.4 and
// 22.4), 512 of 64^2 17.4 and 19.5 (40.6 and 43.1), 4096 of 16^2 17.4 and 29.7 (27.7 and 50.6),
// 16384 of 16^2 57 and 124 (100 and 211).
constexpr int kOneLaunchInstances = 256;

// scratch: 1 + 2 ninstances (+ ninstances nlevels) words: the ticket (0), then (key(0),
// key(+inf)) per instance and key(+inf) per level, as every launch leaves them.
template <typename S>
int launch_stable_dt(const S* state, const PatchDesc* patches, int ndim, const int* chunk_patch,
                     const int* chunk_start, int nchunks, const double* b0, double gamma, unsigned long long* keys,
                     int ninstances, unsigned long long* level_keys, int nlevels, double cfl, double eta, double kappa,
                     const double* inv_dx2_sum, const double* inv_dx2_levels, double* time, const double* end,
                     double* dt, int advance, unsigned long long* scratch, cudaStream_t stream) {
  if (ninstances > kOneLaunchInstances) {
    const int status = launch_rate_chunks<S>(state, patches, 0, ndim, chunk_patch, chunk_start, nchunks, b0, gamma, keys,
                                             ninstances, stream, level_keys, nlevels);
    return status != kOk ? status
                         : launch_finalize_dt(keys, ninstances, cfl, eta, kappa, gamma, inv_dx2_sum, time, end, dt, advance,
                                              stream, level_keys, inv_dx2_levels, nlevels);
  }
  const RateSlots slots{scratch + 1, ninstances, level_keys ? scratch + 1 + 2 * ninstances : nullptr, nlevels, nullptr};
  const StableDt a{cfl, eta, kappa, gamma, inv_dx2_sum, inv_dx2_levels, time, end, dt, advance, keys, level_keys};
  unsigned* ticket = reinterpret_cast<unsigned*>(scratch);
  // up to 8 blocks a chunk while they make at most 4 blocks an SM: a block costs ~3 us besides
  // its cells (work-list look-up, reduction, ticket), which more rounds carry better
  int parts = 8;
  while (parts > 1 && int64_t(nchunks) * parts > 148 * 4) parts /= 2;
  const int grid = max(nchunks * parts, 1);
  if (ndim == 2)
    launch_after(stable_dt_kernel<S, 2>, grid, kRateThreads, 0, stream, state, patches, chunk_patch, chunk_start,
                 nchunks, parts, b0[0], b0[1], b0[2], slots, ticket, a);
  else
    launch_after(stable_dt_kernel<S, 3>, grid, kRateThreads, 0, stream, state, patches, chunk_patch, chunk_start,
                 nchunks, parts, b0[0], b0[1], b0[2], slots, ticket, a);
  return check_launch("stable_dt");
}

template int launch_stable_dt<float>(const float*, const PatchDesc*, int, const int*, const int*, int, const double*,
                                     double, unsigned long long*, int, unsigned long long*, int, double, double,
                                     double, const double*, const double*, double*, const double*, double*, int,
                                     unsigned long long*, cudaStream_t);
template int launch_stable_dt<double>(const double*, const PatchDesc*, int, const int*, const int*, int, const double*,
                                      double, unsigned long long*, int, unsigned long long*, int, double, double,
                                      double, const double*, const double*, double*, const double*, double*, int,
                                      unsigned long long*, cudaStream_t);

}  // namespace wb
