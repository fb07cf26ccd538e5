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
struct PDft<2> {
  static __device__ __forceinline__ void run(Pair *x) {
    const Pair a = x[0], b = x[1];
    x[0] = padd(a, b);
    x[1] = psub(a, b);
  }
};

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

__device__ __forceinline__ void stg_unit(float2 *p, Pair a) {
  asm volatile("st.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a.re), "l"(a.im) : "memory");
}

// Barrier of a group of NT threads: named, or its warp's.
template <int NT>
__device__ __forceinline__ void group_sync(int id) {
  if constexpr (NT == 32)
    __syncwarp();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(NT) : "memory");
}

// Whether any of the group's threads says so, at a barrier of the group.
template <int NT>
__device__ __forceinline__ bool group_any(int id, bool v) {
  if constexpr (NT == 32) return __any_sync(~0u, v);
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %3, 0;\n\t"
      "bar.red.or.pred p, %1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(any)
      : "r"(id), "n"(NT), "r"((uint32_t)v)
      : "memory");
  return any != 0;
}

// Transform of J rows of N = 16 R2 units along the rows and across them, by a group of
// N J / 16 threads with a named barrier of its own, both exchanges in the shared-memory tile.
// A thread holds 16 units; the T = R2 threads of a row are neighbours in one warp, so the
// exchange inside rows needs only warp barriers.
//
// Row stage 1: thread t of a row holds x = t + R2 e (e < 16); its outputs k1, times
// W_N^(t k1), go to slot (k1, t). Row stage 2: butterflies k1 = t + i T read (k1, 0..R2-1);
// outputs k2 are kx = k1 + 16 k2, written to slot kx of the row. Column stage: butterflies
// q = thread + i * threads read slot q of rows 0..J-1. Slot (k1, t) of a row is
// k1 R2 + (t ^ k1's low bits): the writes of a warp (consecutive t) and its reads
// (consecutive k1) both cover all banks. PAD: units between rows, for the landing tile (its
// 8-byte reads span two rows when T < 16).
// (The row exchange through TMEM, as in MidTile, wants a row bit below t in the lane. The
// inverse pass then stores two rows' 64-byte pieces per half warp: 220 us against 195 for 4
// cubes of 256^3; the forward pass, which waits for its copies, gained nothing.)
template <int N_, int J_, int PAD_>
struct OuterTile {
  static constexpr int N = N_, J = J_, PAD = PAD_, R2 = N / 16, U = 16;
  static constexpr int T = N / U;                // threads per row
  static constexpr int NT = N * J / U;           // threads
  static constexpr int B2 = U / R2, B3 = U / J;  // butterflies per thread
  static constexpr int ROWB = (N + PAD) * 16;    // bytes per row
  static constexpr int BYTES = J * ROWB;
  static constexpr int SW = (R2 < 8 ? R2 : 8) - 1;
  static_assert(T <= 32 && T == R2 && U % J == 0, "a row's threads share a warp");

  int t, row, q, barrier;
  uint32_t base, rowb, tw;  // tile; this thread's row; twiddle table (fill_tw)
  // tid: the thread's index in its group of NT threads; id: the group's named barrier.
  __device__ __forceinline__ OuterTile(int tid, int id, uint32_t tw_) {
    t = tid % T;
    row = tid / T;
    q = tid;
    barrier = id;
    tw = tw_ + t * 16;
  }
  __device__ __forceinline__ void at(uint32_t tile_addr) {
    base = tile_addr;
    rowb = tile_addr + row * ROWB;
  }
  __device__ __forceinline__ void sync() const { group_sync<NT>(barrier); }
  // slots: kx of this thread's row; (k1, t) by its writers and its readers; column
  __device__ __forceinline__ uint32_t nat(int x) const { return rowb + x * 16; }
  __device__ __forceinline__ uint32_t ex_w(int k1) const { return rowb + (t ^ (k1 & SW)) * 16 + k1 * (R2 * 16); }
  __device__ __forceinline__ uint32_t ex_r(int i, int tt) const {
    const int k1 = t + i * T;
    return rowb + k1 * (R2 * 16) + (tt ^ (k1 & SW)) * 16;
  }
  __device__ __forceinline__ uint32_t col(int i, int j) const { return base + (q + i * NT) * 16 + j * ROWB; }

  // v[e] = unit t + R2 e of the row on entry; on exit v[i J + j'] = transform at row output
  // q + i NT, column output j'. after_read() runs once the tile's last read is done by this
  // thread.
  template <class F>
  __device__ __forceinline__ void forward(Pair (&v)[U], F &&after_read) const {
    PDft<16>::run(v);
    sts_pair(ex_w(0), v[0]);
#pragma unroll
    for (int k = 1; k < 16; ++k) {
      const Pair w = lds_pair(tw + k * (R2 * 16));
      sts_pair(ex_w(k), pmul_tw(v[k], w.re, w.im));
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
      for (int k = 0; k < R2; ++k) sts_pair(nat(t + i * T + 16 * k), v[i * R2 + k]);
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

  // The mirror, on swapped (im, re) pairs: v[i J + j'] in, v[e] out (unit t + R2 e). The
  // caller has the tile free of readers on entry; after_read() runs once this thread's last
  // read is done.
  template <class F>
  __device__ __forceinline__ void inverse(Pair (&v)[U], F &&after_read) const {
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
      for (int k = 0; k < R2; ++k) v[i * R2 + k] = lds_pair(nat(t + i * T + 16 * k));
    __syncwarp();
#pragma unroll
    for (int i = 0; i < B2; ++i) {
      PDft<R2>::run(v + i * R2);
#pragma unroll
      for (int k = 0; k < R2; ++k) sts_pair(ex_r(i, k), v[i * R2 + k]);
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = lds_pair(ex_w(k));
    after_read();
#pragma unroll
    for (int k = 1; k < 16; ++k) {
      const Pair w = lds_pair(tw + k * (R2 * 16));
      v[k] = pmul_tw(v[k], w.re, w.im);
    }
    PDft<16>::run(v);
  }

  // Row twiddle table into shared memory: entry k1 R2 + t = W_N^(k1 t), both lanes.
  static constexpr int kTwBytes = N * 16;
  static __device__ __forceinline__ void fill_tw(uint32_t tw, const float2 *tw512) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      const float2 w = __ldg(tw512 + ((i / R2) * (i % R2)) * (512 / N));
      sts_pair(tw + i * 16, Pair{pk(w.x, w.x), pk(-w.y, -w.y)});
    }
  }
};

// ------------------------------------------------------------------ exchange through TMEM
// A warp's 32 TMEM lanes x 64 columns as an exchange buffer: what the 32x32b shape stores
// (thread = lane, register = column) the 16x256b shape loads as a matrix fragment (thread
// t: lanes t/4, t/4 + 8 of a half, columns 2 (t % 4) + {0, 1} of every 8), which swaps lane
// bits 4, 3 with column bits 2, 1 and moves lane bits 2..0 up by two. Two such trips swap
// lane bits 4..1 with four register bits: the exchange between the two stages of a row,
// without shared memory. For the 16 warps of an SM it takes 2 x 645 cycles on pipes of their
// own, against 2,048 cycles of the one shared-memory pipe that all exchanges, loads and
// twiddles of a pass share. In the middle pass that pipe was busy 74% of the time, now 60%:
// 4 cubes of 256^3 in 287 us instead of 322 with a filter per cube, 240 instead of 277 with a
// spectrum. Four registers to an instruction: the whole 64 at once, which must be one block
// of registers before and after, spill 290 bytes.
__device__ __forceinline__ void tm_st_rows(uint32_t addr, const uint32_t (&r)[64]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 0u), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 4u), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 8u), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 12u), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 16u), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 20u), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 24u), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 28u), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 32u), "r"(r[32]), "r"(r[33]), "r"(r[34]), "r"(r[35]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 36u), "r"(r[36]), "r"(r[37]), "r"(r[38]), "r"(r[39]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 40u), "r"(r[40]), "r"(r[41]), "r"(r[42]), "r"(r[43]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 44u), "r"(r[44]), "r"(r[45]), "r"(r[46]), "r"(r[47]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 48u), "r"(r[48]), "r"(r[49]), "r"(r[50]), "r"(r[51]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 52u), "r"(r[52]), "r"(r[53]), "r"(r[54]), "r"(r[55]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 56u), "r"(r[56]), "r"(r[57]), "r"(r[58]), "r"(r[59]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + 60u), "r"(r[60]), "r"(r[61]), "r"(r[62]), "r"(r[63]) : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_ld_rows(uint32_t addr, uint32_t (&r)[64]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr + 0u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr + 4u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]) : "r"(addr + 8u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(addr + 12u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]) : "r"(addr + 16u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]) : "r"(addr + 20u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]) : "r"(addr + 24u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]) : "r"(addr + 28u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]) : "r"(addr + 32u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]) : "r"(addr + 36u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]) : "r"(addr + 40u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]) : "r"(addr + 44u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]) : "r"(addr + 48u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]) : "r"(addr + 52u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]) : "r"(addr + 56u) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63]) : "r"(addr + 60u) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_st_frag(uint32_t addr, const uint32_t (&r)[64]) {
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((0u << 16) + 0u)), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((0u << 16) + 8u)), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((0u << 16) + 16u)), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((0u << 16) + 24u)), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((0u << 16) + 32u)), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((0u << 16) + 40u)), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((0u << 16) + 48u)), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((0u << 16) + 56u)), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((16u << 16) + 0u)), "r"(r[32]), "r"(r[33]), "r"(r[34]), "r"(r[35]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((16u << 16) + 8u)), "r"(r[36]), "r"(r[37]), "r"(r[38]), "r"(r[39]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((16u << 16) + 16u)), "r"(r[40]), "r"(r[41]), "r"(r[42]), "r"(r[43]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((16u << 16) + 24u)), "r"(r[44]), "r"(r[45]), "r"(r[46]), "r"(r[47]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((16u << 16) + 32u)), "r"(r[48]), "r"(r[49]), "r"(r[50]), "r"(r[51]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((16u << 16) + 40u)), "r"(r[52]), "r"(r[53]), "r"(r[54]), "r"(r[55]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((16u << 16) + 48u)), "r"(r[56]), "r"(r[57]), "r"(r[58]), "r"(r[59]) : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + ((16u << 16) + 56u)), "r"(r[60]), "r"(r[61]), "r"(r[62]), "r"(r[63]) : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_ld_frag(uint32_t addr, uint32_t (&r)[64]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr + ((0u << 16) + 0u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr + ((0u << 16) + 8u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]) : "r"(addr + ((0u << 16) + 16u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(addr + ((0u << 16) + 24u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]) : "r"(addr + ((0u << 16) + 32u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]) : "r"(addr + ((0u << 16) + 40u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]) : "r"(addr + ((0u << 16) + 48u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]) : "r"(addr + ((0u << 16) + 56u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]) : "r"(addr + ((16u << 16) + 0u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]) : "r"(addr + ((16u << 16) + 8u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]) : "r"(addr + ((16u << 16) + 16u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]) : "r"(addr + ((16u << 16) + 24u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]) : "r"(addr + ((16u << 16) + 32u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]) : "r"(addr + ((16u << 16) + 40u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]) : "r"(addr + ((16u << 16) + 48u)) : "memory");
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63]) : "r"(addr + ((16u << 16) + 56u)) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Where a unit's word (0 re, 1 im; each word's two halves are neighbours) sits on the way.
// k3..k0: bits of the first stage's output index; l4..l1: the lane bits it changes place with.
// First trip: rows-shape column, with (k3 k2) where the fragment shape takes lane bits from.
__host__ __device__ constexpr int tm_col1(int k, int word) {
  return (k >> 2) << 1 | (k >> 1 & 1) << 3 | word << 4 | (k & 1) << 5;
}
// Between the trips, m = (l4 l3 k1 k0): fragment-shape register of the first trip, rows-shape
// column of the second. They differ by the places of l3 and k0 alone, so that the twiddles
// are applied in place, two units at a time where the two change places.
__host__ __device__ constexpr int tm_frag1(int m, int word) {
  return (m >> 3) << 5 | (m & 1) << 4 | word << 3 | (m >> 1 & 1) << 2 | (m >> 2 & 1) << 1;
}
__host__ __device__ constexpr int tm_col2(int m, int word) {
  return (m >> 3) << 5 | (m >> 2 & 1) << 4 | word << 3 | (m & 3) << 1;
}
// Second trip: fragment-shape register of s = (l4 l3 l2 l1).
__host__ __device__ constexpr int tm_frag2(int s, int word) {
  return (s >> 1 & 1) << 5 | (s >> 2) << 3 | word << 2 | (s & 1) << 1;
}
__device__ __forceinline__ void put_pair(uint32_t (&r)[64], int at_re, int at_im, Pair p) {
  r[at_re] = (uint32_t)p.re, r[at_re + 1] = (uint32_t)(p.re >> 32);
  r[at_im] = (uint32_t)p.im, r[at_im + 1] = (uint32_t)(p.im >> 32);
}
__device__ __forceinline__ Pair get_pair(const uint32_t (&r)[64], int at_re, int at_im) {
  return {(f32x2)r[at_re] | (f32x2)r[at_re + 1] << 32, (f32x2)r[at_im] | (f32x2)r[at_im + 1] << 32};
}
// The twiddles between the trips, r from tm_frag1 to tm_col2 order (or back). tw: this lane's
// column of the table.
template <bool BACK>
__device__ __forceinline__ void tm_twiddle(uint32_t (&r)[64], uint32_t tw) {
  auto one = [&](int m) {
    const Pair w = lds_pair(tw + m * 256);
    const Pair p = BACK ? get_pair(r, tm_col2(m, 0), tm_col2(m, 1)) : get_pair(r, tm_frag1(m, 0), tm_frag1(m, 1));
    return pmul_tw(p, w.re, w.im);
  };
  auto put = [&](int m, Pair p) {
    if (BACK)
      put_pair(r, tm_frag1(m, 0), tm_frag1(m, 1), p);
    else
      put_pair(r, tm_col2(m, 0), tm_col2(m, 1), p);
  };
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int l3 = m >> 2 & 1, k0 = m & 1;
    if (l3 == k0) {
      put(m, one(m));
    } else if (l3 == 0) {  // with its partner l3 = 1, k0 = 0
      const int n = m ^ 5;
      const Pair p = one(m), q = one(n);
      put(m, p);
      put(n, q);
    }
  }
}

// Transform of J rows of N = 16 R2 units, C of them interleaved (C independent tiles side by
// side): along the rows and across them (J), by a group of N J C / 16 threads with a named
// barrier of its own. A thread holds 16 units.
//
// Before the row exchange a thread holds units t + R2 e (e < 16) of one row. Its lane is
// (row, t, interleave c): the lowest bit of c, l0, stays in the lane, bits l4..l1 (row, t and
// the rest of c) change place with the first stage's output index k1, by two trips through
// TMEM with the twiddles W_N^(t k1) between them. After it a thread holds, for
// k1 = lane % 16, 16 units indexed by s = (l4 l3 l2 l1): R2 values of t for each of 16 / R2
// (row, interleave) combinations. The
// second stage's outputs kx = k1 + 16 k2 go to the shared-memory tile, where the column
// stage's threads read slot kx of rows 0..J-1.
// A tile slot (row, kx, c) is the row's unit kx C + c with the 16-byte chunk c swizzled by kx
// so that 8 consecutive lanes always cover all banks.
template <int N_, int J_, int C_>
struct MidTile {
  static constexpr int N = N_, J = J_, C = C_, R2 = N / 16, U = 16;
  static constexpr int T = N / U;                 // threads per row and interleaved tile
  static constexpr int NT = N * J * C / U;        // threads
  static constexpr int NTC = NT / C;              // threads per interleaved tile
  static constexpr int B2 = U / R2, B3 = U / J;   // butterflies per thread
  static constexpr int ROWB = N * C * 16;         // bytes per row
  static constexpr int BYTES = J * ROWB;
  static constexpr int HC = C / 2;                // interleaves that l4..l1 hold: lane = (row, t, c)
  static_assert(T * C == 16 && C >= 2, "two rows to a warp");
  static_assert(U % J == 0 && NT % 32 == 0, "16 units per thread");

  int c, t, row, colt, barrier, k1;
  uint32_t base, rowb, tm, tml;  // tile; this thread's row; TMEM columns; twiddle row of this lane
  // tid: the thread's index in its group of NT threads; id: the group's named barrier;
  // tmem: the warp's 64 exchange columns; tw: the twiddle table (fill_tw).
  __device__ __forceinline__ MidTile(int tid, int id, uint32_t tmem, uint32_t tw) {
    const int lane = tid & 31;
    c = tid % C;
    t = (tid / C) % T;
    row = tid / (C * T);
    colt = tid / C;
    barrier = id;
    k1 = lane & 15;
    tm = tmem;
    tml = tw + (uint32_t)((lane >> 3) * 4 + (lane & 3)) * 16;
  }
  __device__ __forceinline__ void at(uint32_t tile_addr) {
    base = tile_addr;
    rowb = tile_addr + row * ROWB + c * 16;
  }
  __device__ __forceinline__ void sync() const { group_sync<NT>(barrier); }
  // Natural unit x of this thread's row as a load left it.
  __device__ __forceinline__ uint32_t nat(int x) const { return rowb + x * (C * 16); }
  // Slot (kx, c) in a row.
  static __device__ __forceinline__ uint32_t slot(int kx, int cc) {
    return (uint32_t)(kx * C + (cc ^ ((kx * C / 8) & (C - 1)))) * 16;
  }
  __device__ __forceinline__ uint32_t col(int i, int j) const { return base + slot(colt + i * NTC, c) + j * ROWB; }
  // After the exchange: unit s of butterfly i's input t, and its row and interleave (l0 is
  // lane bit 4 now).
  static constexpr int unit_of(int i, int tt) {
    return (i / HC) * 8 + tt * HC + i % HC;
  }
  __device__ __forceinline__ uint32_t out(int i, int k2) const {
    const int l0 = (threadIdx.x >> 4) & 1;
    return base + ((row & ~1) + i / HC) * ROWB + slot(k1 + 16 * k2, (i % HC) * 2 + l0);
  }

  // v[e] = unit t + R2 e of the row on entry; on exit v[i J + j'] = transform at row output
  // colt + i NTC, column output j'. The row's shared memory has been read by its warp.
  // after_read() runs once the tile's last read is done by this thread.
  template <class F>
  __device__ __forceinline__ void forward(Pair (&v)[U], F &&after_read) const {
    PDft<16>::run(v);
    if constexpr (R2 == 1) {  // a row is one thread's
#pragma unroll
      for (int k = 0; k < 16; ++k) sts_pair(base + row * ROWB + slot(k, c), v[k]);
    } else {
      uint32_t r[64];
#pragma unroll
      for (int k = 0; k < 16; ++k) put_pair(r, tm_col1(k, 0), tm_col1(k, 1), v[k]);
      __syncwarp();
      tm_st_rows(tm, r);  // lanes (l4 .. l0)
      tm_ld_frag(tm, r);  // lanes (l2 l1 l0 k3 k2)
      tm_twiddle<false>(r, tml);
      tm_st_rows(tm, r);
      tm_ld_frag(tm, r);  // lanes (l0 k3 k2 k1 k0)
#pragma unroll
      for (int i = 0; i < B2; ++i) {
        Pair x[R2];
#pragma unroll
        for (int tt = 0; tt < R2; ++tt) x[tt] = get_pair(r, tm_frag2(unit_of(i, tt), 0), tm_frag2(unit_of(i, tt), 1));
        PDft<R2>::run(x);
#pragma unroll
        for (int k = 0; k < R2; ++k) sts_pair(out(i, k), x[k]);
      }
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

  // The mirror, on swapped (im, re) pairs: v[i J + j'] in, v[e] out (unit t + R2 e). The
  // caller has the tile free of readers on entry; after_read() runs once this thread's last
  // read is done.
  template <class F>
  __device__ __forceinline__ void inverse(Pair (&v)[U], F &&after_read) const {
#pragma unroll
    for (int i = 0; i < B3; ++i) {
      PDft<J>::run(v + i * J);
#pragma unroll
      for (int j = 0; j < J; ++j) sts_pair(col(i, j), v[i * J + j]);
    }
    sync();
    if constexpr (R2 == 1) {
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = lds_pair(base + row * ROWB + slot(k, c));
      after_read();
    } else {
      back_along_rows(v, after_read);
    }
    PDft<16>::run(v);
  }
  template <class F>
  __device__ __forceinline__ void back_along_rows(Pair (&v)[U], F &&after_read) const {
    uint32_t r[64];
#pragma unroll
    for (int i = 0; i < B2; ++i)
#pragma unroll
      for (int k = 0; k < R2; ++k) v[i * R2 + k] = lds_pair(out(i, k));
    after_read();
#pragma unroll
    for (int i = 0; i < B2; ++i) {
      PDft<R2>::run(v + i * R2);
#pragma unroll
      for (int tt = 0; tt < R2; ++tt)
        put_pair(r, tm_frag2(unit_of(i, tt), 0), tm_frag2(unit_of(i, tt), 1), v[i * R2 + tt]);
    }
    __syncwarp();
    tm_st_frag(tm, r);
    tm_ld_rows(tm, r);
    tm_twiddle<true>(r, tml);
    tm_st_frag(tm, r);
    tm_ld_rows(tm, r);
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = get_pair(r, tm_col1(k, 0), tm_col1(k, 1));
  }

  // Twiddle table (4 KB) in shared memory, by a thread's place between the two trips: entry
  // m 16 + q, m = (l4 l3 k1 k0) the register, q = (l2 l1 k3 k2) the lane, holds W_N^(t k) in
  // both lanes of the pair.
  static constexpr int kTwBytes = 256 * 16;
  static __device__ __forceinline__ void fill_tw(uint32_t tw, const float2 *tw512) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
      const int m = i >> 4, q = i & 15;
      const int s = (m >> 2) << 2 | q >> 2, k = (q & 3) << 2 | (m & 3);  // s = (l4 l3 l2 l1)
      const int tt = (s / HC) % R2;
      const float2 w = __ldg(tw512 + tt * k * (512 / N));
      sts_pair(tw + i * 16, Pair{pk(w.x, w.x), pk(-w.y, -w.y)});
    }
  }
};

}  // namespace convgpu
