// Barrier of a cooperative launch (small cubes in one launch).
#pragma once

#include "tma.cuh"

namespace convgpu {

constexpr unsigned kStatusQueueTimeout = 2u;
constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barrier k (k = 1, 2) of a launch waits until slot[0] reaches k * gridDim.x. Both words of
// slot are zero at launch and, by small_grid_leave, again at its end.
// spin: the probe limit, read by the caller at kernel start (dep_wait_limit) so that the
// read stays off the barrier's critical path.
__device__ __forceinline__ bool small_grid_barrier(unsigned *slot, unsigned target, unsigned *status, uint32_t spin) {
  __shared__ int s_ok;
  __syncthreads();  // this block's stores for the level are done
  if (threadIdx.x == 0) {
    __threadfence();  // ... and visible device-wide before the arrival
    atomicAdd(slot, 1u);
    int ok = 0;
    for (uint32_t i = 0; i < spin; ++i) {
      if ((unsigned)ld_acquire(reinterpret_cast<const int *>(slot)) >= target) {
        ok = 1;
        break;
      }
      __nanosleep(32);
    }
    if (!ok && status) atomicOr(status, kStatusQueueTimeout);
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// By every CTA, after its last barrier or the one that gave up (ok: none did): the last to leave
// sets both words back to zero, so that a launch that gave up leaves nothing to the next one
// or to a replay of itself. A barrier that was passed has seen this CTA's arrival; one that
// gave up may not have.
__device__ __forceinline__ void small_grid_leave(unsigned *slot, bool ok) {
  if (threadIdx.x != 0) return;
  if (!ok) __threadfence();
  if (atomicAdd(slot + 1, 1u) != gridDim.x - 1) return;
  atomicExch(slot, 0u);
  atomicExch(slot + 1, 0u);
}

}  // namespace convgpu
