// Fused z pass for N = 512: forward along z, product with a filter, inverse, in persistent
// CTAs that load one tile while they transform another.
//
// A column of 512 points is a radix-2 step and two 256-point transforms, which are the two
// lanes of a pair (tilefft.cuh): unit n holds p(n) + p(n + 256) and (p(n) - p(n + 256))
// W_512^n, and after two radix-16 stages with one exchange between them it holds kz = 2 k and
// 2 k + 1. The product is lane by lane, the inverse the mirror. Against 16 x 16 x 2 stages on
// single values (k_strided_tma, k_zconv_half) that is one exchange less each way and one
// instruction for two values.
//
// HALF: the filter is the half spectrum of a real filter (herm.cuh), transformed along x and
// y only. A group serves two signal tiles of 8 columns: A, columns x0.. of row y, and B,
// columns N - x0 - 8.. of row -y. The filter of B's column c is the conjugate, point by
// point of z, of the filter's column x0 + 8 - c of row y, so with B's values conjugated when
// they are loaded and stored both tiles use one filter tile, of 9 columns (10 for the copy's
// alignment), which is transformed once, by the same threads, before the signals. Otherwise a
// group serves one tile of 8 columns and a filter tile of as many: transformed along z
// already, or here (FZ).
//
// Tiles are claimed in order (claims: a counter, zero at launch, counts those after the
// first of every group): SMs differ by a third in how long a tile takes them, and with a
// fixed share of the tiles the fastest were done after 70% of the pass.
//
// Bound by HBM and the latency of a tile's chain of stages: a tile's filter is loaded during
// the inverse of the tile before, its signals during that one's last stage and the filter's
// transform, and two (three) groups per SM fill each other's gaps. One 512^3 cube, us: HALF
// 617 (2.7 GB: 4.4 TB/s; its loads and stores alone take 502, 64-byte rows 2 MB apart), where
// k_zconv_half took 691 and the filter's own z pass 204; a full spectrum 690 instead of 770,
// with its z transform 730 instead of 840. Five warps of their own for the filters, which
// leaves 96 registers a thread: 693 with HALF.
#pragma once

#include "herm.cuh"
#include "passes.cuh"
#include "tilefft.cuh"
#include "tilestream.cuh"

namespace convgpu {

// C: columns per tile; FC: columns of a filter tile; NT: threads of a group; G: groups per
// CTA, one CTA per SM (104 KB a group with HALF, else 64 KB).
template <bool HALF>
struct ZPairShape {
  static constexpr int N = 512, U = 256, C = 8, FC = HALF ? C + 2 : C, TILES = HALF ? 2 : 1, NT = 128 * TILES,
                       G = HALF ? 2 : 3, GROUPS = (HALF ? N / 2 : N) / C;
  static constexpr int TB = N * C * 8, SB = TILES * TB, FB = N * FC * 8, PITCH = SB + FB;
  static constexpr int kSmem = 2048 + G * PITCH + 2 * U * 16;
};

// The 16 x 16 transform of a column of units by 16 threads, thread t of them; ROWB: bytes
// between units. Slot of (k1, t) between the stages is 16 k1 + t.
template <int ROWB>
struct UnitColumn {
  uint32_t base, tw, tw2;  // the column's unit 0; W_256^(t k1) at k1 16 + t; radix-2 twiddles, by n
  int t;
  __device__ __forceinline__ uint32_t at(int n) const { return base + n * ROWB; }
  // Radix-2 step of units t + 16 e, from points n and n + 256 of a column of complex values
  // `pitch` bytes apart; sgn -1 conjugates.
  __device__ __forceinline__ void load(Pair (&v)[16], uint32_t points, int pitch, float sgn) const {
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int n = t + 16 * e;
      const float2 p = lds_f2(points + n * pitch), q = lds_f2(points + (n + 256) * pitch);
      v[e] = {pk(p.x + q.x, p.x - q.x), pk(sgn * (p.y + q.y), sgn * (p.y - q.y))};
    }
  }
  // Units t + 16 e -> first stage's outputs k1, twiddled.
  __device__ __forceinline__ void stage1(Pair (&v)[16]) const {
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const Pair w = lds_pair(tw2 + (t + 16 * e) * 16);
      v[e] = pmul_tw(v[e], w.re, w.im);
    }
    PDft<16>::run(v);
#pragma unroll
    for (int k = 1; k < 16; ++k) {
      const Pair w = lds_pair(tw + (k * 16 + t) * 16);
      v[k] = pmul_tw(v[k], w.re, w.im);
    }
  }
  __device__ __forceinline__ void write1(const Pair (&v)[16]) const {
#pragma unroll
    for (int k = 0; k < 16; ++k) sts_pair(at(16 * k + t), v[k]);
  }
  __device__ __forceinline__ void read1(Pair (&v)[16]) const {
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = lds_pair(at(16 * k + t));
  }
  // This thread's 16 slots as the second stage's butterfly k1 = t: (k1, 0..15).
  __device__ __forceinline__ void write2(const Pair (&v)[16]) const {
#pragma unroll
    for (int k = 0; k < 16; ++k) sts_pair(at(16 * t + k), v[k]);
  }
  __device__ __forceinline__ void read2(Pair (&v)[16]) const {
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = lds_pair(at(16 * t + k));
  }
};

// A kernel, not a memset: a memset may be queued on a copy engine behind large transfers.
static __global__ void k_zpair_clear(unsigned *claims) { *claims = 0u; }

// msig: the signals, box {C, 1, 256}; mfilt: the filter's columns, box {FC, 1, 256}.
template <bool HALF, bool FZ>
__global__ void __launch_bounds__(ZPairShape<HALF>::NT *ZPairShape<HALF>::G, 1)
    k_zpair(const __grid_constant__ CUtensorMap msig, const __grid_constant__ CUtensorMap mfilt, PassArgs a, int nvol,
            unsigned *claims) {
  using S = ZPairShape<HALF>;
  constexpr int N = S::N, C = S::C, FC = S::FC, NT = S::NT, G = S::G;
  static_assert(FZ || !HALF, "a half spectrum comes untransformed along z");
  extern __shared__ __align__(128) unsigned char smraw[];
  const uint32_t sm = smem_u32(smraw), tw = sm + 2048 + G * S::PITCH, tw2 = tw + S::U * 16;
  // loads of signals and of filters; load n of either is this CTA's n-th tile, group n % G's
  const TpStream<G, G> ss{sm, sm + 2048, (uint32_t)S::PITCH}, fs{sm + 1024, sm + 2048 + S::SB, (uint32_t)S::PITCH};
  const int g = threadIdx.x / NT, tid = threadIdx.x % NT;
  const int ntiles = nvol * N * S::GROUPS;
  auto load_filter = [&](int n, int w) {  // by one thread; says which tile (below zero: none) load n is
    fs.set_tile(n, w < ntiles ? w : -1);
    if (w >= ntiles) {
      mbar_arrive(fs.full(n));
      return;
    }
    const int r = w % (N * S::GROUPS), y = r / S::GROUPS, x0 = r % S::GROUPS * C;
    const int z0 = a.filt_vol_elems ? w / (N * S::GROUPS) * N : 0;
    mbar_arrive_expect_tx(fs.full(n), S::FB);
    tma_load_3d(fs.buf(n), &mfilt, x0, y, z0, fs.full(n));
    tma_load_3d(fs.buf(n) + S::FB / 2, &mfilt, x0, y, z0 + N / 2, fs.full(n));
  };
  auto load_signal = [&](int n, int w) {
    if (w >= ntiles) return;
    const int r = w % (N * S::GROUPS), y = r / S::GROUPS, x0 = r % S::GROUPS * C, z0 = w / (N * S::GROUPS) * N;
    mbar_arrive_expect_tx(ss.full(n), S::SB);
#pragma unroll
    for (int i = 0; i < S::TILES; ++i) {
      const int x = i ? N - x0 - C : x0, yy = i ? (N - y) & (N - 1) : y;
      tma_load_3d(ss.buf(n) + i * S::TB, &msig, x, yy, z0, ss.full(n));
      tma_load_3d(ss.buf(n) + i * S::TB + S::TB / 2, &msig, x, yy, z0 + N / 2, ss.full(n));
    }
  };
  if (threadIdx.x == 0) {
    ss.init();
    fs.init();
    for (int n = 0; n < G; ++n) {
      load_filter(n, blockIdx.x * G + n);
      load_signal(n, blockIdx.x * G + n);
    }
  }
  for (int i = threadIdx.x; i < S::U; i += blockDim.x) {
    const float2 w = __ldg(a.tw512 + (i >> 4) * (i & 15) * 2), u = __ldg(a.tw512 + i);
    sts_pair(tw + i * 16, Pair{pk(w.x, w.x), pk(-w.y, -w.y)});
    sts_pair(tw2 + i * 16, Pair{pk(1.f, u.x), pk(0.f, -u.y)});
  }
  __syncthreads();
  const int half = tid / 128, c = tid % C, t = tid % 128 / C;  // tile, column, thread of the column
  const float sgn = half ? -1.f : 1.f;
  const int fcol = half ? C - c : c;
  auto group_barrier = [&] { group_sync<NT>(1 + g); };
  auto tile_barrier = [&] { group_sync<128>(HALF ? 1 + G + g * 2 + half : 1 + g); };
  bool ok = true;
  Pair v[16];
  for (int n = g;; n += G) {
    const uint32_t fbuf = fs.buf(n), sbuf = ss.buf(n) + half * S::TB;
    // the whole group carries on or stops
    if (group_any<NT>(1 + g, !fs.wait(n) || !ok)) {
      ok = false;
      break;
    }
    const int w = fs.tile(n);
    if (w < 0) break;
    int next = 0;  // the group's next tile, claimed ahead of its use below
    if (tid == 0) next = (int)(gridDim.x * G + atomicAdd(claims, 1u));
    if constexpr (FZ) {
      const bool mine = tid < FC * 16;  // whole warps
      const UnitColumn<FC * 16> f{fbuf + (uint32_t)(tid % FC) * 16, tw, tw2, tid / FC};
      if (mine) {
        f.load(v, fbuf + (uint32_t)(tid % FC) * 8, FC * 8, 1.f);
        f.stage1(v);
      }
      group_barrier();
      if (mine) f.write1(v);
      group_barrier();
      if (mine) {
        f.read2(v);
        PDft<16>::run(v);
      }
      group_barrier();
      if (mine) f.write1(v);  // output k = t + 16 k2 to slot k
    }
    const UnitColumn<C * 16> s{sbuf + (uint32_t)c * 16, tw, tw2, t};
    ok &= ss.wait(n);
    s.load(v, sbuf + (uint32_t)c * 8, C * 8, sgn);
    s.stage1(v);
    group_barrier();
    s.write1(v);
    tile_barrier();
    s.read2(v);
    PDft<16>::run(v);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      Pair f;
      if constexpr (FZ) {
        f = lds_pair(fbuf + (uint32_t)((t + 16 * k) * FC + fcol) * 16);
      } else {
        const uint32_t at = fbuf + (uint32_t)(2 * (t + 16 * k) * FC + fcol) * 8;
        const float2 p = lds_f2(at), q = lds_f2(at + FC * 8);
        f = {pk(p.x, q.x), pk(p.y, q.y)};
      }
      v[k] = pswap(pmul(v[k], f));
    }
    PDft<16>::run(v);
    s.write2(v);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    group_barrier();
    if (tid == 0) load_filter(n + G, fs.marked() ? ntiles : next);
    s.read1(v);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    group_barrier();
    if (tid == 0) load_signal(n + G, fs.tile(n + G) < 0 ? ntiles : next);
#pragma unroll
    for (int k = 1; k < 16; ++k) {
      const Pair w = lds_pair(tw + (k * 16 + t) * 16);
      v[k] = pmul_tw(v[k], w.re, w.im);
    }
    PDft<16>::run(v);
    const int r = w % (N * S::GROUPS), y = r / S::GROUPS, x0 = r % S::GROUPS * C;
    float2 *o = a.dst + (long long)(w / (N * S::GROUPS)) * N * N * N +
                (long long)(half ? (N - y) & (N - 1) : y) * N + (half ? N - x0 - C : x0) + c;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const Pair u = lds_pair(tw2 + (t + 16 * e) * 16);
      const Pair p = pmul_tw(v[e], u.re, u.im);  // swapped: re holds im
      const float sy = sgn * a.scale;
      float2 *oz = o + (long long)(t + 16 * e) * N * N;
      oz[0] = make_float2((lo_of(p.im) + hi_of(p.im)) * a.scale, (lo_of(p.re) + hi_of(p.re)) * sy);
      oz[256ll * N * N] = make_float2((lo_of(p.im) - hi_of(p.im)) * a.scale, (lo_of(p.re) - hi_of(p.re)) * sy);
    }
  }
  if (!ok) {
    tp_gave_up(ss, a.status);
    tp_gave_up(fs, a.status);
  }
}

// x pass of a real filter into the half layout (the first half_pitch(512) values of a row's
// spectrum): two rows a, b as one complex row z = a + i b, whose spectrum Z gives
// A(k) = (Z(k) + conj Z(-k)) / 2 and B(k) = (Z(k) - conj Z(-k)) / 2i. 16 threads transform a
// pair of rows in place in shared memory, as above; a warp's two pairs are its own, from
// the load to the stores, so warps run apart. Bound by HBM: 1.1 GB in 159 us at 512^3 (one
// row at a time, k_rows_real, 317).
struct RowsRealPair {
  static constexpr int N = 512, U = 256, WARPS = 4, W = half_pitch(N);
  static constexpr int PAIR = 2 * N * 4 + 64;  // bytes of a pair of rows; the pad keeps a warp's two on other banks
  static constexpr int kSmem = 128 + WARPS * 2 * PAIR + 2 * U * 16;
  static constexpr int kRows = WARPS * 4;
};
static __global__ void __launch_bounds__(RowsRealPair::WARPS * 32, 4) k_rows_real_pair(PassArgs a) {
  using S = RowsRealPair;
  constexpr int N = S::N, U = S::U;
  extern __shared__ __align__(128) unsigned char smraw[];
  const uint32_t sm = smem_u32(smraw), tw = sm + 128 + S::WARPS * 2 * S::PAIR, tw2 = tw + U * 16;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, t = lane % 16;
  const uint32_t bar = sm + warp * 8, rows = sm + 128 + warp * 2 * S::PAIR, mine = rows + lane / 16 * S::PAIR;
  const long long row0 = ((long long)blockIdx.x * S::WARPS + warp) * 4;
  if (lane == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
    mbar_arrive_expect_tx(bar, 4 * N * 4);
    const float *src = reinterpret_cast<const float *>(a.src) + row0 * N;
    bulk_load(rows, src, 2 * N * 4, bar);
    bulk_load(rows + S::PAIR, src + 2 * N, 2 * N * 4, bar);
  }
  for (int i = threadIdx.x; i < U; i += blockDim.x) {
    const float2 w = __ldg(a.tw512 + (i >> 4) * (i & 15) * 2), u = __ldg(a.tw512 + i);
    sts_pair(tw + i * 16, Pair{pk(w.x, w.x), pk(-w.y, -w.y)});
    sts_pair(tw2 + i * 16, Pair{pk(1.f, u.x), pk(0.f, -u.y)});
  }
  __syncthreads();
  const bool ok = mbar_wait_bounded(bar, 0);
  __syncwarp();
  if (!ok && a.status) atomicOr(a.status, kStatusTmaTimeout);
  Pair v[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const uint32_t at = mine + (t + 16 * e) * 4;
    const float pa = lds_f(at), qa = lds_f(at + U * 4), pb = lds_f(at + N * 4), qb = lds_f(at + N * 4 + U * 4);
    const Pair w = lds_pair(tw2 + (t + 16 * e) * 16);
    v[e] = pmul_tw(Pair{pk(pa + qa, pa - qa), pk(pb + qb, pb - qb)}, w.re, w.im);
  }
  PDft<16>::run(v);
  __syncwarp();
  // slot of (k1, t): 16 k1 + (t ^ k1), all banks for either side
  sts_pair(mine + t * 16, v[0]);
#pragma unroll
  for (int k = 1; k < 16; ++k) {
    const Pair w = lds_pair(tw + (k * 16 + t) * 16);
    sts_pair(mine + (16 * k + (t ^ k)) * 16, pmul_tw(v[k], w.re, w.im));
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = lds_pair(mine + (16 * t + (k ^ t)) * 16);
  PDft<16>::run(v);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 16; ++k)  // Z(2 j) and Z(2 j + 1), j = t + 16 k, as complex values side by side
    sts_pair(mine + (t + 16 * k) * 16, Pair{pk(lo_of(v[k].re), lo_of(v[k].im)), pk(hi_of(v[k].re), hi_of(v[k].im))});
  __syncwarp();
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    float2 *o = a.dst + (row0 + 2 * p) * S::W;
    for (int k = lane; k < S::W; k += 32) {
      const float2 z = lds_f2(rows + p * S::PAIR + k * 8), m = lds_f2(rows + p * S::PAIR + ((N - k) & (N - 1)) * 8);
      o[k] = make_float2(0.5f * (z.x + m.x), 0.5f * (z.y - m.y));
      o[S::W + k] = make_float2(0.5f * (z.y + m.y), 0.5f * (m.x - z.x));
    }
  }
}

}  // namespace convgpu
