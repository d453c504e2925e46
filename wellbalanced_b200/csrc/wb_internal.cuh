// Internal helpers shared by the CUDA translation units: launch checks, the library's
// last-error text, exact order-independent max/min reductions through integer keys.
#pragma once

#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>

namespace wb {

// Status codes of the C ABI (also in include/wellbalanced_b200.h).
enum Status : int {
  kOk = 0,
  kBadArgument = -1,
  kCudaError = -2,
  kUnsupported = -3,
  kTooLarge = -4,
};

void set_error(const char* fmt, ...);
const char* last_error();

inline int check_launch(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s: CUDA launch failed: %s", what, cudaGetErrorString(e));
    return kCudaError;
  }
  return kOk;
}

// A step is a chain of launches that are short on small grids and refined hierarchies, so the
// kernels of a step overlap their launch with the kernel before: launched by `launch_after`
// (programmatic stream serialization), each starts with `after_previous`, which waits until
// the kernel before it in the stream has finished and its memory is visible, and then lets
// the next one be set up. No kernel reads or writes global memory before that call, so the
// order of all accesses is that of plain launches. That holds for coherent loads only: the
// compiler may read what a `const T* __restrict__` kernel parameter points to through the
// read-only path, or before the call, and the kernel before may still be writing it. So such
// a parameter is for tables that no launch writes (patches, op lists); the pools, the dt, the
// flux register and the boundary fluxes are not marked so. B200: the refined sheet (25 launches a step)
// 542 -> 476 us for two steps, 256^2 float64 (3 a step) 214 -> 200 us for four. A launch that is
// refused leaves its error for the `check_launch` after it.
template <typename... P, typename... A>
inline void launch_after(void (*kernel)(P...), int64_t grid, int threads, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(unsigned(grid));
  config.blockDim = dim3(unsigned(threads));
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute = {};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  cudaLaunchKernelEx(&config, kernel, P(args)...);
}

__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Order-preserving map of a double onto uint64: a < b  <=>  key(a) < key(b) (non-NaN).
__device__ __forceinline__ unsigned long long double_to_key(double x) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__host__ __device__ __forceinline__ double key_to_double_bits(unsigned long long k) {
  const unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  double out;
  memcpy(&out, &b, sizeof(out));
  return out;
}

__device__ __forceinline__ double key_to_double(unsigned long long k) {
  const unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double(static_cast<long long>(b));
}

// keys[0] = key(0) (running max of a non-negative rate), keys[1] = key(+inf) (running min)
__global__ void init_keys_kernel(unsigned long long* keys);

// Block-wide max of `largest` and min of `smallest`, one atomic per warp; the min also
// into *level_min when given.
__device__ __forceinline__ void block_reduce_keys(double largest, double smallest,
                                                  unsigned long long* keys,
                                                  unsigned long long* level_min = nullptr) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    largest = fmax(largest, __shfl_xor_sync(0xffffffffu, largest, o));
    smallest = fmin(smallest, __shfl_xor_sync(0xffffffffu, smallest, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&keys[0], double_to_key(largest));
    atomicMin(&keys[1], double_to_key(smallest));
    if (level_min) atomicMin(level_min, double_to_key(smallest));
  }
}

}  // namespace wb
