// The stream of tile loads of a persistent CTA (twopass.cuh, pairs512.cuh).
#pragma once

#include "tma.cuh"

namespace convgpu {

// Buffers and barriers of a CTA's stream of loads. Load n belongs to group n % G and lands
// in buffer n % B; load n + B takes the buffer once that group is done with it. Its "full"
// barrier is the group's own, one of 4 in turn: a group waits for its loads in order, so a
// parity is never read a phase early (a barrier per buffer serves several groups, and one
// that is ahead would take the phase before its load's for its own), and a barrier is never
// armed while its earlier copy is outstanding: load n + 4 G is issued once load n + 4 G - B
// is consumed, by the group that consumed load n + B before, which took load n's buffer.
template <int B, int G>
struct TpStream {
  static_assert(2 * B % G == 0 && 4 * G - B >= B, "barriers per group");
  uint32_t bar, tiles, pitch;
  __device__ __forceinline__ uint32_t full(int n) const { return bar + ((n % G) * 4 + (n / G) % 4) * 8; }
  __device__ __forceinline__ uint32_t buf(int n) const { return tiles + (n % B) * pitch; }
  // The outer passes' tile of load n (below zero: none is left), written before its barrier is
  // armed and read after the wait.
  __device__ __forceinline__ uint32_t tile_slot(int n) const { return bar + 720 + ((n % G) * 4 + (n / G) % 4) * 4; }
  __device__ __forceinline__ void set_tile(int n, int w) const {
    asm volatile("st.shared.s32 [%0], %1;" ::"r"(tile_slot(n)), "r"(w) : "memory");
  }
  __device__ __forceinline__ int tile(int n) const {
    int w;
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(w) : "r"(tile_slot(n)) : "memory");
    return w;
  }
  // A bounded wait that gave up marks the CTA: it carries on with what its buffers hold
  // (wrong output, reported through the status word), waits no more and loads no more.
  __device__ __forceinline__ uint32_t mark() const { return bar + 704; }
  __device__ __forceinline__ bool marked() const {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(mark()) : "memory");
    return v != 0;
  }
  __device__ __forceinline__ bool wait_on(uint32_t b, uint32_t parity) const {
    bool ok = mbar_try_wait(b, parity);
    if (!ok && !marked()) {
      ok = mbar_wait_bounded(b, parity);
      if (!ok) asm volatile("st.shared.u32 [%0], %1;" ::"r"(mark()), "r"(1u) : "memory");
    }
    __syncwarp();
    return ok;
  }
  // By all lanes of each warp.
  __device__ __forceinline__ bool wait(int n) const { return wait_on(full(n), (uint32_t)(n / (4 * G)) & 1u); }
  // By thread 0, before the barriers are used.
  __device__ __forceinline__ void init() const {
    for (int i = 0; i < 4 * G; ++i) mbar_init(bar + i * 8, 1);
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(mark()), "r"(0u) : "memory");
    mbar_fence_init();
  }
};

// After a wait that gave up: reports it, and lets copies still in flight land before the
// CTA leaves. A barrier's current phase is the one whose parity is not complete.
template <int B, int G>
__device__ __forceinline__ void tp_gave_up(const TpStream<B, G> &st, unsigned *status) {
  if (status) atomicOr(status, kStatusTmaTimeout);
  for (int b = 0; b < 4 * G; ++b) {
    const uint32_t parity = mbar_try_wait(st.bar + b * 8, 0) ? 1u : 0u;
    for (int i = 0; i < 1 << 14; ++i)
      if (mbar_try_wait(st.bar + b * 8, parity)) break;
  }
}

}  // namespace convgpu
