// A step's launches from one call: the host hands over a list of C-ABI calls (function code and
// argument slots) that it put together once per layout, and `wb_run_launches` issues them in
// order on the caller's stream, `repeat` times. From Python each call costs ~8 us (argument
// conversion, pointer look-ups), more than the small kernels of a 2D step run; from here ~2.
// B200: a 32^2 float64 step (with one status read instead of two) 120 -> 94 us, the refined
// sheet of 25 launches a step 563 -> 535 us for two steps.
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>
#include <utility>

#include "wb_internal.cuh"
#include "wellbalanced_b200.h"

using namespace wb;

namespace {

// the event calls of a side stream's fork and join, and clearing a counter
int record_event(void* event, void* stream) {
  const cudaError_t e = cudaEventRecord(static_cast<cudaEvent_t>(event), static_cast<cudaStream_t>(stream));
  if (e == cudaSuccess) return kOk;
  set_error("record_event: %s", cudaGetErrorString(e));
  return kCudaError;
}
int wait_event(void* event, void* stream) {
  const cudaError_t e = cudaStreamWaitEvent(static_cast<cudaStream_t>(stream), static_cast<cudaEvent_t>(event), 0);
  if (e == cudaSuccess) return kOk;
  set_error("wait_event: %s", cudaGetErrorString(e));
  return kCudaError;
}
int clear_bytes(void* ptr, int64_t bytes, void* stream) {
  const cudaError_t e = cudaMemsetAsync(ptr, 0, size_t(bytes), static_cast<cudaStream_t>(stream));
  if (e == cudaSuccess) return kOk;
  set_error("clear_bytes: %s", cudaGetErrorString(e));
  return kCudaError;
}

// An argument from its 8-byte slot: integers and pointers as they are, doubles by their bits.
template <typename T>
T slot(int64_t v) {
  return static_cast<T>(v);
}
template <>
double slot<double>(int64_t v) {
  double d;
  std::memcpy(&d, &v, sizeof(d));
  return d;
}
template <typename T>
struct Slot {
  static T get(int64_t v) { return slot<T>(v); }
};
template <typename T>
struct Slot<T*> {
  static T* get(int64_t v) { return reinterpret_cast<T*>(v); }
};

// the last argument of every function is the stream
template <typename... A, size_t... I>
int call(int (*f)(A...), const int64_t* a, void* stream, std::index_sequence<I...>) {
  return f((I + 1 == sizeof...(A) ? Slot<A>::get(reinterpret_cast<int64_t>(stream)) : Slot<A>::get(a[I]))...);
}
template <auto F, typename... A>
int run_with(int (*f)(A...), const int64_t* a, void* stream) {
  return call(f, a, stream, std::index_sequence_for<A...>{});
}
template <auto F>
int run(const int64_t* a, void* stream) {
  return run_with<F>(F, a, stream);
}

struct Entry {
  const char* name;
  int (*run)(const int64_t*, void*);
};

const Entry kEntries[] = {
    {"wb_stage2d_tiled", run<wb_stage2d_tiled>},
    {"wb_stage2d_physics", run<wb_stage2d_physics>},
    {"wb_stage3d_tiled", run<wb_stage3d_tiled>},
    {"wb_stage3d_physics", run<wb_stage3d_physics>},
    {"wb_stable_dt", run<wb_stable_dt>},
    {"wb_copy_ops", run<wb_copy_ops>},
    {"wb_interp_ops", run<wb_interp_ops>},
    {"wb_fill_ops", run<wb_fill_ops>},
    {"wb_restrict_ops", run<wb_restrict_ops>},
    {"wb_face_flux_ops", run<wb_face_flux_ops>},
    {"wb_face_flux_ops_physics", run<wb_face_flux_ops_physics>},
    {"wb_face_flux_ops_staged", run<wb_face_flux_ops_staged>},
    {"wb_reflux_apply", run<wb_reflux_apply>},
    {"record_event", run<record_event>},
    {"wait_event", run<wait_event>},
    {"clear_bytes", run<clear_bytes>},
};
constexpr int kCount = int(sizeof(kEntries) / sizeof(kEntries[0]));

}  // namespace

extern "C" int wb_launch_code(const char* name) {
  set_error("");
  for (int i = 0; name && i < kCount; ++i)
    if (std::strcmp(name, kEntries[i].name) == 0) return i;
  set_error("launch_code: no launch named %s", name ? name : "(null)");
  return kBadArgument;
}

extern "C" int wb_run_launches(const void* launches, int count, int repeat, void* stream) {
  set_error("");
  if (count < 0 || repeat < 0 || (count > 0 && !launches)) {
    set_error("run_launches: bad list");
    return kBadArgument;
  }
  const wb_launch* list = static_cast<const wb_launch*>(launches);
  for (int i = 0; i < count; ++i)
    if (list[i].code < 0 || list[i].code >= kCount) {
      set_error("run_launches: entry %d has no launch code %d", i, int(list[i].code));
      return kBadArgument;
    }
  for (int r = 0; r < repeat; ++r)
    for (int i = 0; i < count; ++i) {
      void* s = list[i].own_stream ? reinterpret_cast<void*>(list[i].stream) : stream;
      const int status = kEntries[list[i].code].run(list[i].args, s);
      if (status != kOk) return status;
    }
  return kOk;
}
