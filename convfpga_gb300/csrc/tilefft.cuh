// Building blocks of the two-pass 3D transform (twopass.cuh): arithmetic on pairs of
// complex values, radix-4/8/16 DFTs on them, and the tile transform that a CTA runs on
// rows x columns of such pairs through shared memory.
//
// A pair holds two independent complex values, one per lane of two packed FP32 registers:
// re = (re0, re1), im = (im0, im1). Every addition, multiplication and FMA of a transform is
// then one packed two-lane instruction (sm_100 and later) for two values, a rotation by -i
// is a renaming of registers, and a twiddle is loaded once for both. In memory a pair is a
// 16-byte unit {re0, re1, im0, im1}, one 128-bit access. Against the one-value form
// (fft_core.cuh: packed additions only, scalar multiplications) a radix-16 stage of two
// values takes 144 + 60 instructions instead of 2 x (120 + 60), which matters because the
// passes of the three-axis form issue on about half of their cycles.
//
// The inverse transform is swap(re, im) -> forward -> swap, as everywhere in this library;
// on pairs the swap is a renaming as well.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "tma.cuh"

namespace convgpu {

using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pk(float lo, float hi) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float lo_of(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_of(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 neg2(f32x2 a) { return a ^ 0x8000000080000000ull; }

// Two complex values, lane-wise.
struct Pair {
  f32x2 re, im;
};
__device__ __forceinline__ Pair padd(Pair a, Pair b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ Pair psub(Pair a, Pair b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
__device__ __forceinline__ Pair pswap(Pair a) { return {a.im, a.re}; }
// a * (c - i s), c and s per lane.
__device__ __forceinline__ Pair pmul_tw(Pair a, f32x2 c, f32x2 s) {
  return {fma2(a.im, s, mul2(a.re, c)), fma2(a.im, c, mul2(a.re, neg2(s)))};
}
// a * b
__device__ __forceinline__ Pair pmul(Pair a, Pair b) {
  return {fma2(a.im, neg2(b.im), mul2(a.re, b.re)), fma2(a.im, b.re, mul2(a.re, b.im))};
}

// In-place forward 4-point DFT, natural order.
__device__ __forceinline__ void pdft4(Pair &a, Pair &b, Pair &c, Pair &d) {
  const Pair t0 = padd(a, c), t1 = psub(a, c), t2 = padd(b, d), t3 = psub(b, d);
  a = padd(t0, t2);
  c = psub(t0, t2);
  b = {add2(t1.re, t3.im), sub2(t1.im, t3.re)};
  d = {sub2(t1.re, t3.im), add2(t1.im, t3.re)};
}

// Forward DFT of R points at x[0], x[STRIDE], ...: natural order in and out.
template <int R>
struct PDft;

template <>
struct PDft<4> {
  static __device__ __forceinline__ void run(Pair *x) { pdft4(x[0], x[1], x[2], x[3]); }
};

template <>
struct PDft<8> {
  // Two 4-point DFTs (even, odd inputs) and a radix-2 step whose eighth-turn factors
  // sqrt(1/2)(1 -+ i) are an add and a subtract with the scale folded into the final FMAs.
  static __device__ __forceinline__ void run(Pair *x) {
    const f32x2 r = pk(0.70710678118654752440f, 0.70710678118654752440f), nr = neg2(r);
    Pair e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
    pdft4(e[0], e[1], e[2], e[3]);
    pdft4(o[0], o[1], o[2], o[3]);
    x[0] = padd(e[0], o[0]);
    x[4] = psub(e[0], o[0]);
    const Pair p = {add2(o[1].re, o[1].im), sub2(o[1].im, o[1].re)};  // W8 o1 = r p
    x[1] = {fma2(p.re, r, e[1].re), fma2(p.im, r, e[1].im)};
    x[5] = {fma2(p.re, nr, e[1].re), fma2(p.im, nr, e[1].im)};
    x[2] = {add2(e[2].re, o[2].im), sub2(e[2].im, o[2].re)};  // -i o2
    x[6] = {sub2(e[2].re, o[2].im), add2(e[2].im, o[2].re)};
    const Pair q = {sub2(o[3].re, o[3].im), add2(o[3].re, o[3].im)};  // W8^3 o3 = -r q
    x[3] = {fma2(q.re, nr, e[3].re), fma2(q.im, nr, e[3].im)};
    x[7] = {fma2(q.re, r, e[3].re), fma2(q.im, r, e[3].im)};
  }
};

template <>
struct PDft<16> {
  // 4 x 4: four 4-point DFTs over x[i + 4m], then four over i with the twiddles W16^(ik),
  // each written C (1 -+ i T) or C (T -+ i) with C = cos(pi/8), T = tan(pi/8), so that C is
  // folded into the last additions as FMAs: 144 packed operations.
  static __device__ __forceinline__ void run(Pair *x) {
    const f32x2 r = pk(0.70710678118654752440f, 0.70710678118654752440f), nr = neg2(r);
    const f32x2 C = pk(0.92387953251128675613f, 0.92387953251128675613f), nC = neg2(C);
    const f32x2 T = pk(0.41421356237309504880f, 0.41421356237309504880f), nT = neg2(T);
#pragma unroll
    for (int i = 0; i < 4; ++i) pdft4(x[i], x[i + 4], x[i + 8], x[i + 12]);
    Pair y[16];
    {  // k = 0: no twiddles
      pdft4(x[0], x[1], x[2], x[3]);
      y[0] = x[0], y[4] = x[1], y[8] = x[2], y[12] = x[3];
    }
    {  // k = 1: 1, C(1 - iT), r(1 - i), C(T - i)
      const Pair a = x[4], b = x[5], c = x[6], d = x[7];
      const Pair g = {add2(c.re, c.im), sub2(c.im, c.re)};
      const Pair t0 = {fma2(g.re, r, a.re), fma2(g.im, r, a.im)}, t1 = {fma2(g.re, nr, a.re), fma2(g.im, nr, a.im)};
      const Pair p = {fma2(b.im, T, b.re), fma2(b.re, nT, b.im)};
      const Pair q = {fma2(d.re, T, d.im), fma2(d.im, T, neg2(d.re))};
      const Pair s = padd(p, q), m = psub(p, q);
      y[1] = {fma2(s.re, C, t0.re), fma2(s.im, C, t0.im)};
      y[9] = {fma2(s.re, nC, t0.re), fma2(s.im, nC, t0.im)};
      y[5] = {fma2(m.im, C, t1.re), fma2(m.re, nC, t1.im)};
      y[13] = {fma2(m.im, nC, t1.re), fma2(m.re, C, t1.im)};
    }
    {  // k = 2: 1, r(1 - i), -i, -r(1 + i)
      const Pair a = x[8], b = x[9], c = x[10], d = x[11];
      const Pair t0 = {add2(a.re, c.im), sub2(a.im, c.re)}, t1 = {sub2(a.re, c.im), add2(a.im, c.re)};
      const Pair p = {add2(b.re, b.im), sub2(b.im, b.re)};
      const Pair q = {sub2(d.re, d.im), add2(d.re, d.im)};
      const Pair s = psub(p, q), m = padd(p, q);
      y[2] = {fma2(s.re, r, t0.re), fma2(s.im, r, t0.im)};
      y[10] = {fma2(s.re, nr, t0.re), fma2(s.im, nr, t0.im)};
      y[6] = {fma2(m.im, r, t1.re), fma2(m.re, nr, t1.im)};
      y[14] = {fma2(m.im, nr, t1.re), fma2(m.re, r, t1.im)};
    }
    {  // k = 3: 1, C(T - i), -r(1 + i), -C(1 - iT)
      const Pair a = x[12], b = x[13], c = x[14], d = x[15];
      const Pair g = {sub2(c.re, c.im), add2(c.re, c.im)};
      const Pair t0 = {fma2(g.re, nr, a.re), fma2(g.im, nr, a.im)}, t1 = {fma2(g.re, r, a.re), fma2(g.im, r, a.im)};
      const Pair p = {fma2(b.re, T, b.im), fma2(b.im, T, neg2(b.re))};
      const Pair q = {fma2(d.im, T, d.re), fma2(d.re, nT, d.im)};
      const Pair s = psub(p, q), m = padd(p, q);
      y[3] = {fma2(s.re, C, t0.re), fma2(s.im, C, t0.im)};
      y[11] = {fma2(s.re, nC, t0.re), fma2(s.im, nC, t0.im)};
      y[7] = {fma2(m.im, C, t1.re), fma2(m.re, nC, t1.im)};
      y[15] = {fma2(m.im, nC, t1.re), fma2(m.re, C, t1.im)};
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = y[k];
  }
};

// 16-byte units in shared memory, by 32-bit address.
__device__ __forceinline__ Pair lds_pair(uint32_t a) {
  Pair p;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(p.re), "=l"(p.im) : "r"(a) : "memory");
  return p;
}
__device__ __forceinline__ void sts_pair(uint32_t a, Pair p) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(p.re), "l"(p.im) : "memory");
}
__device__ __forceinline__ float2 lds_f2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float lds_f(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// Radix split of a row length: R1 first, R2 second.
template <int N>
struct RowSplit;
template <> struct RowSplit<256> { static constexpr int R1 = 16, R2 = 16; };
template <> struct RowSplit<128> { static constexpr int R1 = 16, R2 = 8; };
template <> struct RowSplit<64> { static constexpr int R1 = 8, R2 = 8; };
template <> struct RowSplit<32> { static constexpr int R1 = 8, R2 = 4; };
template <> struct RowSplit<16> { static constexpr int R1 = 4, R2 = 4; };

// Transform of J rows of N units, C of them interleaved (C independent tiles side by side):
// along the rows (N = R1 * R2) and across them (J), by a group of N J C / 16 threads with a
// named barrier of its own. A thread holds 16 units; the N / 16 threads of a row and its C
// interleaved tiles are neighbours in one warp, so the exchange inside rows needs only warp
// barriers and only the one across rows a group barrier.
//
// Row stage 1: thread t of a row holds x = t + i T + R2 e (butterfly i, e < R1); its outputs
// k1, times W_N^(t k1), go to slot (k1, t). Row stage 2: butterflies k1 = t + i T read
// (k1, 0..R2-1); outputs k2 are kx = k1 + R1 k2, written to slot kx of the row. Column
// stage: butterflies q = thread + i * threads read slot q of rows 0..J-1.
// Slot (k1, t) of a row is k1 R2 + (t ^ k1's low bits): the writes of a warp (consecutive t)
// and its reads (consecutive k1) both cover all banks. PAD: units between rows, for the
// landing tile of the first pass (its 8-byte reads span several rows when T < 16).
template <int N_, int J_, int C_, int PAD_ = 0>
struct Tile {
  static constexpr int N = N_, J = J_, C = C_, PAD = PAD_;
  static constexpr int R1 = RowSplit<N>::R1, R2 = RowSplit<N>::R2, U = 16;
  static constexpr int T = N / U;                 // threads per row and interleaved tile
  static constexpr int NT = N * J * C / U;        // threads
  static constexpr int NTC = NT / C;              // threads per interleaved tile
  static constexpr int B1 = U / R1, B2 = U / R2, B3 = U / J;
  static constexpr int ROWB = (N * C + PAD) * 16;  // bytes per row
  static constexpr int BYTES = J * ROWB;
  static constexpr int SW = (R2 < 8 ? R2 : 8) - 1;
  static_assert(T >= 1 && C * T <= 32, "a row's threads share a warp");
  static_assert(U % J == 0 && T * B1 == R2 && T * B2 == R1, "16 units per thread");

  int c, t, row, colt, barrier;
  uint32_t base, rowb;  // tile; this thread's row
  // tid: the thread's index in its group of NT threads; id: the group's named barrier.
  __device__ __forceinline__ Tile(int tid, int id) {
    c = tid % C;
    t = (tid / C) % T;
    row = tid / (C * T);
    colt = tid / C;
    barrier = id;
  }
  __device__ __forceinline__ void at(uint32_t tile_addr) {
    base = tile_addr;
    rowb = tile_addr + row * ROWB + c * 16;
  }
  __device__ __forceinline__ void sync() const {
    asm volatile("bar.sync %0, %1;" ::"r"(barrier), "n"(NT) : "memory");
  }
  __device__ __forceinline__ int t1(int i) const { return t + i * T; }
  // slots: natural unit x of this thread's row; exchange slots; column unit
  __device__ __forceinline__ uint32_t nat(int x) const { return rowb + x * (C * 16); }
  __device__ __forceinline__ uint32_t ex_w(int k1, int i) const {  // k1 constant
    return rowb + ((t + i * T) ^ (k1 & SW)) * (C * 16) + k1 * (R2 * C * 16);
  }
  __device__ __forceinline__ uint32_t ex_r(int i, int tt) const {  // tt constant
    const int k1 = t + i * T;
    return rowb + k1 * (R2 * C * 16) + (tt ^ (k1 & SW)) * (C * 16);
  }
  __device__ __forceinline__ uint32_t col(int i, int j) const {
    return base + c * 16 + (colt + i * NTC) * (C * 16) + j * ROWB;
  }

  // v[i R1 + e] = unit t1(i) + R2 e of the row on entry; on exit v[i J + j'] = transform at
  // row output colt + i NTC, column output j'. tw: table {c, c, s, s} of W_N^(k1 t) at
  // k1 R2 + t. after_read() runs once the tile's last read is done by this thread.
  template <class F>
  __device__ __forceinline__ void forward(Pair (&v)[U], uint32_t tw, F &&after_read) const {
#pragma unroll
    for (int i = 0; i < B1; ++i) {
      PDft<R1>::run(v + i * R1);
      sts_pair(ex_w(0, i), v[i * R1]);
#pragma unroll
      for (int k = 1; k < R1; ++k) {
        const Pair w = lds_pair(tw + (k * R2 + t1(i)) * 16);
        sts_pair(ex_w(k, i), pmul_tw(v[i * R1 + k], w.re, w.im));
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < B2; ++i)
#pragma unroll
      for (int k = 0; k < R2; ++k) v[i * R2 + k] = lds_pair(ex_r(i, k));
    __syncwarp();
#pragma unroll
    for (int i = 0; i < B2; ++i) {
      PDft<R2>::run(v + i * R2);
#pragma unroll
      for (int k = 0; k < R2; ++k) sts_pair(nat(t1(i) + R1 * k), v[i * R2 + k]);
    }
    sync();
#pragma unroll
    for (int i = 0; i < B3; ++i)
#pragma unroll
      for (int j = 0; j < J; ++j) v[i * J + j] = lds_pair(col(i, j));
    after_read();
#pragma unroll
    for (int i = 0; i < B3; ++i) PDft<J>::run(v + i * J);
  }

  // The mirror, on swapped (im, re) pairs: v[i J + j'] in, v[i R1 + e] out (unit
  // t1(i) + R2 e). The caller has the tile free of readers on entry; after_read() runs once
  // this thread's last read is done.
  template <class F>
  __device__ __forceinline__ void inverse(Pair (&v)[U], uint32_t tw, F &&after_read) const {
#pragma unroll
    for (int i = 0; i < B3; ++i) {
      PDft<J>::run(v + i * J);
#pragma unroll
      for (int j = 0; j < J; ++j) sts_pair(col(i, j), v[i * J + j]);
    }
    sync();
#pragma unroll
    for (int i = 0; i < B2; ++i)
#pragma unroll
      for (int k = 0; k < R2; ++k) v[i * R2 + k] = lds_pair(nat(t1(i) + R1 * k));
    __syncwarp();
#pragma unroll
    for (int i = 0; i < B2; ++i) {
      PDft<R2>::run(v + i * R2);
#pragma unroll
      for (int k = 0; k < R2; ++k) sts_pair(ex_r(i, k), v[i * R2 + k]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < B1; ++i) {
#pragma unroll
      for (int k = 0; k < R1; ++k) v[i * R1 + k] = lds_pair(ex_w(k, i));
    }
    after_read();
#pragma unroll
    for (int i = 0; i < B1; ++i) {
#pragma unroll
      for (int k = 1; k < R1; ++k) {
        const Pair w = lds_pair(tw + (k * R2 + t1(i)) * 16);
        v[i * R1 + k] = pmul_tw(v[i * R1 + k], w.re, w.im);
      }
      PDft<R1>::run(v + i * R1);
    }
  }

  // Row twiddle table into shared memory: entry k1 R2 + t = W_N^(k1 t), both lanes.
  static __device__ __forceinline__ void fill_tw(uint32_t tw, const float2 *tw512) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      const float2 w = __ldg(tw512 + ((i / R2) * (i % R2)) * (512 / N));
      sts_pair(tw + i * 16, Pair{pk(w.x, w.x), pk(-w.y, -w.y)});
    }
  }
};

}  // namespace convgpu
