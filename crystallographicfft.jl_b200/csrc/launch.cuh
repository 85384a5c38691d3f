// Launch helpers shared by the kernel translation units: programmatic dependent launch and
// error conversion.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>
#include <string>
#include <utility>

#include "cfft_internal.h"

namespace cfft {
namespace {

// Programmatic dependent launch: wait until the previous kernel of the stream has
// completed and its writes are visible (a no-op when the kernel was launched without
// the attribute), then let the next kernel of the stream start launching.  Called in
// every kernel that launch_k starts, before any access to memory that a kernel writes.
// Loads of the plan's constant tables may come before it: they are then in flight while the
// previous kernel finishes.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

constexpr int kSMs = 148;  // B200: the unit of the launch-size rules

// Programmatic dependent launch of the fast-path kernels (off with CFFT_PDL=0): each
// kernel of a lane may launch while its predecessor in the stream is finishing, and
// waits for it in hardware (griddepcontrol.wait, pdl_enter) before touching memory that
// another kernel writes.
inline bool pdl_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("CFFT_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}
// First failure of a launch_k launch on this thread since fast_unit_launch last read it.
inline cudaError_t& launch_error() {
  static thread_local cudaError_t e = cudaSuccess;
  return e;
}
template <typename... KArgs, typename... Args>
inline void launch_k(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  if (pdl_enabled()) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, std::forward<Args>(args)...);
    if (e != cudaSuccess && launch_error() == cudaSuccess) launch_error() = e;
  } else {
    k<<<grid, block, smem, st>>>(std::forward<Args>(args)...);
  }
}

inline Status fast_cuda(cudaError_t e, const char* what, std::string* err) {
  if (e == cudaSuccess) return Status::kOk;
  *err = std::string(what) + ": " + cudaGetErrorString(e);
  return Status::kCuda;
}

}  // namespace
}  // namespace cfft
