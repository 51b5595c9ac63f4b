// Shared definitions of the n3 CUDA library (sm_100a).
//
// State layout in HBM and shared memory: the reference's interleaved slot
// layout (src/no_three_75/accelerated.py:18-24, src/no_three_75/tempering.py:38):
// slot s = 2*row + layer, row(s) = s >> 1, column = cols[s].  A state of an
// n x n grid has m = 2n slots.  Rows are implicit, so a state is m columns.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/n3.h"

namespace n3 {

constexpr int kMaxN = N3_MAX_N;        // 75: 150 slots, the reference's bound
constexpr int kMaxM = 2 * N3_MAX_N;    // 150
constexpr int kLutW = 2 * kMaxN - 1;   // dy in [-(kMaxN-1), kMaxN-1]
constexpr int kLutSize = kMaxN * kLutW;  // dx in [0, kMaxN-1]

// Device error word bits (written by kernels, read by the host after a sync).
enum : uint32_t {
  kErrColumnRange = 1u << 0,   // a column outside [0, n)
  kErrDuplicate = 1u << 1,     // two points of one row coincide
  kErrMismatch = 1u << 2,      // determinant and slope counts disagree
  kErrTimeout = 1u << 3,       // a bounded wait gave up
  kErrAudit = 1u << 4,         // incremental energy differs from a full recompute
  kErrCapacity = 1u << 5,      // an output list was longer than the caller's capacity
};

// First in a kernel launched by launch_chained: lets the next kernel of the chain be
// brought onto the SMs, then waits until the one before has finished and its
// writes are visible.  Nothing before it in the kernel may touch memory or hold
// tensor memory.  Without effect in a kernel launched otherwise.  Such a kernel
// lives while the ones before it still write, so it reads nothing of theirs through
// the read-only path: no __ldg and no `const T* __restrict__` in its parameters or in
// what it passes them to (its outputs may be restricted); the wait orders ordinary
// loads only.
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ int warp_sum(int v) { return __reduce_add_sync(0xffffffffu, v); }

}  // namespace n3

// Host-side helpers shared by the .cu files (defined in capi.cu).
namespace n3host {
int set_error(int code, const char* fmt, ...);
int check_launch(const char* what);
int ensure_device_tables();
int sm_count();
int allow_smem(const void* kernel, size_t bytes);

// A launch whose blocks may be brought onto the SMs while the kernel before it in
// the stream still runs (programmatic stream serialization), for short kernels
// that follow each other; the kernel begins with n3::chain_begin().  It saves 1 to
// 2 us per launch: a training step of seven 70 -> 60 us, a learned step of five
// 107 -> 99 us, a beam generation of five 188 -> 183 us.
template <class... Params, class... Args>
int launch_chained(const char* what, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                   Args... args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = st;
  config.attrs = &attr;
  config.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
  if (e != cudaSuccess) return set_error(N3_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  return check_launch(what);
}
}  // namespace n3host

#define N3_TRY(expr)                      \
  do {                                    \
    const int n3_rc_ = (expr);            \
    if (n3_rc_ != N3_OK) return n3_rc_;   \
  } while (0)
