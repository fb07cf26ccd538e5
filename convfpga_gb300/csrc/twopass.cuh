// A 3D convolution in tiles instead of axes: the whole forward transform is two passes over
// memory and so is the inverse, with the product between them.
//
// A cube of N^3 points is cut so that each pass transforms as many points as a CTA holds.
// With y = y0 + R j (R = N / J) and planes zz and zz + N/2 together:
//   k_tp_fwd   the radix-2 step of z across the two planes, all of x, and J points of y: a
//              tile of J rows x N points x 2 planes (64 KB at N = 256);
//   k_tp_mid   the remaining R points of y and N/2 points of z: a tile of R rows x N/2 points
//              x C columns; forward, product with the filter's spectrum, inverse;
//   k_tp_inv   the mirror of k_tp_fwd.
// Against one pass per axis (or x and y together through an L2-resident ring, xyl2.cuh) a
// signal crosses memory three times as in the ring form (16 + 24 + 16 N^3 bytes with its
// filter operand), but no CTA waits for another, the twelve radix-16 steps of forward and
// inverse need eight exchanges instead of twelve, and nothing goes through a ring in L2.
//
// The two planes' values are the two lanes of a pair (tilefft.cuh). The radix-2 step turns
// them into the even and odd half of z, which stay independent, so a pair is transformed
// lane by lane from the first load to the last store:
//   lane 0: p(zz) + p(zz + N/2), lane 1: (p(zz) - p(zz + N/2)) W_N^zz.
// The intermediate array ("tile order") holds a cube as tiles of k_tp_mid, contiguous:
//   tile g N + kx (g = j' / C), in it unit (y0 N/2 + zz) C + j' % C
// so a thread of k_tp_fwd, which ends with all j' of one kx, stores runs of C 16-byte units,
// and k_tp_mid reads and writes whole tiles. Scattering runs of 32 bytes costs nothing: a
// tile scatter of 4 cubes of 256^3 measured 169 us with 32-byte runs and 164 us with 64-byte
// runs, a plain copy 170 us (neighbouring tiles in flight fill each other's lines in L2).
// A spectrum in tile order holds, in tile (g, kx), unit (k2 N/2 + kz') C + c: the pairs
// (kz = 2 kz' and 2 kz' + 1) at ky = g C + c + J k2.
//
// Persistent CTAs take tiles in order through a few buffers in shared memory. The reference
// streams each axis through its own engine with transposes between (kernels/conv3D.cl:71-420).
#pragma once

#include "gridsync.cuh"
#include "tilefft.cuh"
#include "tilestream.cuh"

namespace convgpu {

// Per-size shape: J rows of the outer tile, C interleaved columns of the middle tile, G
// groups of threads per CTA (one CTA per SM), B tile buffers. A group transforms one tile at
// a time; the other B - G buffers are in flight, so a group finds its next tile landed.
//   256: 64 KB tiles, 2 groups of 256 threads x 128 registers, 3 buffers.
//   128: 32 KB tiles, 4 groups of 128 threads, 6 buffers. 64: 16 KB, 8 groups of 64, 12
//   buffers. 32: 8 KB, 16 groups of a warp, 24 buffers.
// One CTA of 16 compute warps per SM, since a thread holds a tile's 16 pairs (64 registers).
// Measured, us: 4 cubes of 256^3: k_tp_fwd 177 and k_tp_inv 180 (1.07 GB each: 6.0 TB/s; two
// CTAs of one tile each, loaded and stored from registers, took 215 and 276), k_tp_mid with
// a filter per cube 285 (1.6 GB: 5.6 TB/s), so 808 for a batch with its filters, against
// 1,083 for the L2-staged x+y passes and the fused z pass. At N = 64 a pass of 33 cubes takes
// 30 to 39: 128 KB of tiles per SM take some 6.3 us whatever the size, and 33 cubes are 3.5
// rounds of that.
template <int N>
struct TpShape;
template <>
struct TpShape<256> {
  static constexpr int J = 16, C = 2, PAD = 0, G = 2, B = 3;
};
template <>
struct TpShape<128> {
  static constexpr int J = 16, C = 4, PAD = 4, G = 4, B = 6;
};
template <>
struct TpShape<64> {
  static constexpr int J = 16, C = 8, PAD = 4, G = 8, B = 12;
};
template <>
struct TpShape<32> {
  static constexpr int J = 16, C = 16, PAD = 2, G = 16, B = 24;
};
// Units of a run that one TMA box row holds (128 bytes at most, for the swizzle).
template <int N>
constexpr int kTpBox = TpShape<N>::C < 8 ? TpShape<N>::C : 8;

// The filter operand of k_tp_mid.
enum TpMode : int {
  TP_PAIR = 0,      // filter in tile order, not yet transformed along the rest of y and z
  TP_SPECTRUM = 1,  // filter spectrum in tile order
  TP_FWD = 2,       // no filter: the forward half alone (makes a spectrum)
};

struct TpArgs {
  const float2 *src;   // k_tp_fwd: cubes; k_tp_mid, k_tp_inv: cubes in tile order
  const float2 *src2;  // k_tp_fwd: cubes `first`.. come from here (and go to the second map)
  int first;
  float2 *dst;
  const float2 *filt;  // k_tp_mid
  long long src_vol, dst_vol, filt_vol;  // elements between cubes (0: one for all)
  int nvol;
  float scale;  // k_tp_inv
  const float2 *tw512;
  unsigned *status;
  // Cubes at unrelated addresses (device arrays of nvol pointers and tensor maps), else null.
  const CUtensorMap *maps;  // k_tp_fwd: dst; k_tp_inv: src
  const float2 *const *srcs;
  float2 *const *dsts;
  const float2 *const *filts;
  __device__ __forceinline__ const float2 *src_of(int v) const { return srcs ? srcs[v] : src + v * src_vol; }
  __device__ __forceinline__ float2 *dst_of(int v) const { return dsts ? dsts[v] : dst + v * dst_vol; }
  __device__ __forceinline__ const float2 *filt_of(int v) const { return filts ? filts[v] : filt + v * filt_vol; }
};

template <int N>
using TpOuterTile = OuterTile<N, TpShape<N>::J, TpShape<N>::PAD>;
template <int N>
using TpMidTile = MidTile<N / 2, N / TpShape<N>::J, TpShape<N>::C>;

template <int N>
constexpr int kTpThreads = TpOuterTile<N>::NT *TpShape<N>::G;

// Bytes between the tile buffers: the largest tile (the outer one's rows may be padded), a
// multiple of 1 KB.
template <int N>
constexpr int kTpBuf = (TpOuterTile<N>::BYTES + 1023) / 1024 * 1024;

// Shared memory: barriers and TMEM slot (1 KB, keeps the tiles aligned), tiles, row
// twiddles, then the outer passes' step twiddles (two sets of J per group) and the linear
// table W_N^j.
template <int N>
constexpr int tp_outer_smem() {
  return 1024 + TpShape<N>::B * kTpBuf<N> + TpOuterTile<N>::kTwBytes + TpShape<N>::G * 2 * TpShape<N>::J * 16 + N * 8;
}
template <int N>
constexpr int tp_mid_smem() {
  return 1024 + TpShape<N>::B * kTpBuf<N> + TpMidTile<N>::kTwBytes;
}

// Step twiddles of outer tile (y0, zz): entry j' = {W_N^(y0 j'), W_N^(y0 j' + zz)} as
// {c0, c1, s0, s1}; written by the group's first J threads into one of its two sets, since
// slow threads may still read the previous tile's.
template <int N>
__device__ __forceinline__ void tp_step_tw(uint32_t utw, uint32_t lin, int tid, int y0, int zz) {
  if (tid < TpShape<N>::J) {
    const float2 a = lds_f2(lin + ((y0 * tid) & (N - 1)) * 8), b = lds_f2(lin + ((y0 * tid + zz) & (N - 1)) * 8);
    sts_pair(utw + tid * 16, Pair{pk(a.x, b.x), pk(-a.y, -b.y)});
  }
}

// Programmatic dependent launch: a CTA may start once every CTA of the kernel before it in the
// stream has started to end, fills its tables and sets up its barriers, and touches nothing
// that another kernel writes before tp_grid_wait(). It hides the launch and the set-up of
// every pass but the first: 17 cubes of 32^3 21.8 us instead of 30.8, one of 128^3 44.7 instead
// of 52.2, three of 256^3 529 instead of 538. (Letting the next kernel in from the start, launch_dependents, changed nothing there
// and cost 4 cubes of 256^3 with their filters 909 us instead of 835.)
__device__ __forceinline__ void tp_grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// TMEM of a CTA (warp 1 allocates and frees): 64 columns per warp that shares a lane group,
// for the row exchange, and in the middle pass as many again for the filter's values.
template <int COLS>
__device__ __forceinline__ uint32_t tp_tmem_alloc(uint32_t slot) {
  if (threadIdx.x / 32 == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "n"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(slot) : "memory");
  return tmem;
}
template <int COLS>
__device__ __forceinline__ void tp_tmem_free(uint32_t tmem) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (threadIdx.x / 32 == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(COLS));
}
// This warp's 64 columns of block b.
__device__ __forceinline__ uint32_t tp_tmem_warp(uint32_t tmem, int b) {
  const int w = threadIdx.x >> 5;
  return tmem + ((uint32_t)(32 * (w & 3)) << 16) + (uint32_t)(256 * b + 64 * (w >> 2));
}

// Tiles of the outer passes at N = 128 and 256 are claimed in order, after each CTA's first
// ones, not dealt out: runs of 32 or 64 bytes of neighbouring tiles share cache lines, which
// leave L2 half filled (about 20 us after the first write) if CTAs with a fixed share of the
// tiles drift apart. A forward pass of 32 cubes of 256^3 then took 123 us a cube and filter
// where one of 8 took 91, and the inverse 51 a cube; claimed 85 and 42. At N = 32 and 64 runs
// are whole lines, and the claims of so many small tiles cost more than they give (17 cubes
// of 32^3 64 us instead of 25, before those took their stores from the tile's own buffer). One
// counter per size and pass (kernels of one size and pass never run side by side); every tile claims one successor,
// so the claim that counts the last tile is the last there is and sets it back to zero. The
// middle pass between them zeroes both as well, for after a pass that gave up.
__device__ unsigned g_tp_claims[4];
template <int N>
constexpr bool kTpClaims = N >= 128;
template <int N>
constexpr bool kTpStager = N >= 64;  // k_tp_fwd: a warp of its own stores the tiles
template <int N>
__device__ __forceinline__ unsigned *tp_claims(int pass) {
  return g_tp_claims + (N == 256 ? 2 : 0) + pass;
}
// Tile of a CTA's load n (ntiles or above: none is left), claimed by one thread when one of
// the launch's tiles is begun; the first `dealt` tiles of the launch are the CTAs' own, tile
// blockIdx + n gridDim, and so are all of a short launch, over before CTAs drift.
template <int N>
__device__ __forceinline__ int tp_claim(int pass, int n, int dealt, int ntiles) {
  if (ntiles < 32 * (int)gridDim.x) return (int)(blockIdx.x + n * gridDim.x);
  const unsigned k = atomicAdd(tp_claims<N>(pass), 1u);
  if (k == (unsigned)ntiles - 1u) atomicExch(tp_claims<N>(pass), 0u);
  return dealt + (int)k;
}

__device__ __forceinline__ void tma_store_3d(const CUtensorMap *m, uint32_t src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(src), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}

// Byte offset of unit c of kx's run in a staged (or landed) box: boxes of N runs of C units,
// 16-byte chunks swizzled as the tensor map says (32, 64 or 128 bytes), so that neighbouring
// kx cover all banks.
template <int C>
__device__ __forceinline__ uint32_t tp_run_off(int kx, int c) {
  return (uint32_t)(kx * C + (c ^ ((kx * C / 8) & (C - 1)))) * 16;
}

// Forward outer pass. REAL: the first a.first cubes hold N^3 floats each (real filters), the
// others complex values. mdst: the destination in
// tile order, dims (2 C values of a run, tiles, runs of a tile), box (2 C, N, 1), for the
// first a.first cubes, mdst2 for the others (a filter and its signals in one launch).
//
// N = 64 to 256: every group has a buffer of its own, where its loads land and its exchanges
// happen; the next load is issued when the columns are in registers. Outputs are staged in
// the other S = B - G buffers, which the groups take in turn, and a further warp stores them:
// 2,048 runs of 32 bytes keep the TMA unit for about 1.8 us, which the tile's own buffer does
// not wait for. (Stores from registers, one run per thread, hold the LSU pipe for 1.4 cycles
// a run, 80% of the pass: 215 us for 4 cubes of 256^3. Staged in the tile's own buffer 195,
// this 187, 177 with claimed tiles.)
// N = 32: outputs are staged in the tile's own buffer and stored by the group; the buffer
// takes its next load during the group's next tile. (One warp storing for 16 groups holds
// them up: 17 cubes under one filter 24.6 us instead of 21.8. At N = 64 it does not: 100
// cubes 239 us instead of 258.)
template <int N>
constexpr int kTpFwdThreads = kTpThreads<N> + (kTpStager<N> ? 32 : 0);

template <int N, bool REAL>
__global__ void __launch_bounds__(kTpFwdThreads<N>, 1)
    k_tp_fwd(const __grid_constant__ CUtensorMap mdst, const __grid_constant__ CUtensorMap mdst2, TpArgs a) {
  using TT = TpOuterTile<N>;
  using S = TpShape<N>;
  constexpr int J = TT::J, R = N / J, C = S::C, H = N / 2, G = S::G, B = S::B, SB = B - G,
                BX = kTpBox<N>;
  static_assert(G % SB == 0, "the groups take the staging buffers in turn");
  extern __shared__ __align__(1024) unsigned char smraw[];
  const uint32_t sm = smem_u32(smraw);
  const TpStream<B, G> st{sm, sm + 1024, (uint32_t)kTpBuf<N>};
  const uint32_t tw = sm + 1024 + B * kTpBuf<N>, utw0 = tw + TT::kTwBytes, lin = utw0 + G * 2 * J * 16;
  const int g = threadIdx.x / TT::NT, tid = threadIdx.x % TT::NT;
  const int ntiles = a.nvol * R * H;
  constexpr bool kClaims = kTpClaims<N>, kStager = kTpStager<N>;
  const int mine = kClaims ? 0 : ((int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0);
  // staged[s]: the group whose turn it is has staged its tile in buffer G + s;
  // grant[g]: the buffer of group g's next turn has been stored (a group's own, so its waits
  // are in order). Turn n is group n % G's and buffer G + n % SB's.
  const uint32_t staged = sm + 512, grant = sm + 576;
  static_assert(G <= 16 && SB <= 8, "barriers in the first KB");
  auto real = [&](int vol) { return REAL && vol < a.first; };  // this cube's rows are floats
  auto load = [&](int n, int w) {  // by one warp: 2 J row copies, row (j, plane) at j ROWB + plane N 8
    const int lane = threadIdx.x & 31;
    if (w >= ntiles) {
      if (lane == 0) {
        st.set_tile(n, -1);
        mbar_arrive(st.full(n));
      }
      return;
    }
    const int vol = w / (R * H), r = w % (R * H), y0 = r / H, zz = r % H;
    // src_vol counts values, complex or float
    const uint32_t row = real(vol) ? N * 4 : N * 8;
    const char *src = a.srcs ? (const char *)a.srcs[vol]
                             : (vol < a.first ? (const char *)a.src + vol * a.src_vol * (REAL ? 4 : 8)
                                              : (const char *)a.src2 + (vol - a.first) * a.src_vol * 8);
    if (lane == 0) {
      st.set_tile(n, w);
      mbar_arrive_expect_tx(st.full(n), 2 * J * row);
    }
    __syncwarp();
    for (int i = lane; i < 2 * J; i += 32) {
      const int j = i >> 1, z = zz + (i & 1) * H;
      bulk_load(st.buf(kStager ? n % G : n) + j * TT::ROWB + (i & 1) * (N * 8), src + ((long long)z * N + y0 + R * j) * row, row,
                st.full(n));
    }
  };
  auto store = [&](uint32_t buf, int w) {  // by one thread: the staged tile's runs
    const int vol = w / (R * H), r = w % (R * H);
    const CUtensorMap *m = a.maps ? a.maps + vol : (vol < a.first ? &mdst : &mdst2);
    const int mvol = a.maps ? 0 : (vol < a.first ? vol : vol - a.first);
    if (a.maps) tensormap_acquire(m);
#pragma unroll
    for (int k = 0; k < J / BX; ++k)  // box k: units k BX .. of the runs of column group k BX / C
      tma_store_3d(m, buf + k * (N * BX * 16), 0, (mvol * (J / C) + k * BX / C) * N, r * (C / BX) + k % (C / BX));
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  };
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) {
      for (int s = 0; s < SB; ++s) mbar_init(staged + s * 8, TT::NT);
      for (int i = 0; i < G; ++i) mbar_init(grant + i * 8, 1);
      st.init();
    }
    __syncwarp();
    tp_grid_wait();
    for (int n = 0; n < (kClaims ? G : min(kStager ? G : B, mine)); ++n) load(n, blockIdx.x + n * gridDim.x);
  }
  TT::fill_tw(tw, a.tw512);
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const float2 w = __ldg(a.tw512 + i * (512 / N));
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(lin + i * 8), "f"(w.x), "f"(w.y) : "memory");
  }
  tp_grid_wait();
  __syncthreads();
  bool ok = true;
  if (kStager && !kClaims && g == G) {  // the storing warp, turns known
    for (int n = 0; n < mine; ++n) {
      const int s = n % SB;
      ok &= st.wait_on(staged + s * 8, (uint32_t)(n / SB) & 1u);
      if (tid == 0) {
        store(st.buf(G + s), blockIdx.x + n * gridDim.x);
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        if (n + SB < mine) mbar_arrive(grant + (n + SB) % G * 8);
      }
      __syncwarp();
    }
    if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    if (!ok) tp_gave_up(st, a.status);
    return;
  }
  if (kClaims && g == G) {  // the storing warp
    unsigned alive = (1u << G) - 1u;
    int done[SB] = {};  // phases of each staging buffer
    for (int n0 = 0; alive; n0 += SB) {
#pragma unroll
      for (int s = 0; s < SB; ++s) {
        const int n = n0 + s, turn = n % G;
        if (!(alive >> turn & 1u)) continue;
        ok &= st.wait(n);  // the turn's tile is known
        const bool none = ok && st.tile(n) < 0;
        if (!__any_sync(~0u, none)) ok &= st.wait_on(staged + s * 8, (uint32_t)(done[s]++) & 1u);
        if (__any_sync(~0u, !ok || st.marked())) {  // a wait gave up: no more stores
          ok = false;
          alive = 0;
          break;
        }
        const int w = st.tile(n);
        if (w < 0) {
          alive &= ~(1u << turn);
        } else if (tid == 0) {
          store(st.buf(G + s), w);
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
        if (tid == 0) {  // the buffer's next turn that is still taken
          for (int m = n + SB; m < n + SB + G; m += SB)
            if (alive >> (m % G) & 1u) {
              mbar_arrive(grant + m % G * 8);
              break;
            }
        }
        __syncwarp();
      }
    }
    if (tid == 0) {
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    if (!ok) tp_gave_up(st, a.status);
    return;
  }
  TT tt(tid, 1 + g, tw);
  int set = 0, drain = -1;  // drain: the load whose buffer the group's last store reads (N = 32)
  for (int n = g; kClaims || n < mine; n += G) {
    int w = blockIdx.x + n * gridDim.x;
    if constexpr (kClaims) {
      // the whole group carries on or stops
      if (group_any<TT::NT>(1 + g, !st.wait(n) || !ok)) {
        ok = false;
        break;
      }
      w = st.tile(n);
      if (w < 0) break;  // nothing left; the storing warp sees it too and passes the turn on
      tt.at(st.buf(g));
    } else {
      ok &= st.wait(n);
      tt.at(st.buf(kStager ? g : n));
    }
    const int r = w % (R * H), y0 = r / H, zz = r % H;
    const uint32_t utw = utw0 + (g * 2 + set) * (J * 16);
    tp_step_tw<N>(utw, lin, tid, y0, zz);
    int next = 0;  // the group's next tile, claimed ahead of its use below
    if (kClaims && tid == 0) next = tp_claim<N>(0, n + G, gridDim.x * G, ntiles);
    Pair v[16];
    if (real(w / (R * H))) {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int x = tt.t + TT::R2 * e;
        const float p = lds_f(tt.rowb + x * 4), q = lds_f(tt.rowb + N * 8 + x * 4);
        v[e] = {pk(p + q, p - q), 0ull};
      }
    } else {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int x = tt.t + TT::R2 * e;
        const float2 p = lds_f2(tt.rowb + x * 8), q = lds_f2(tt.rowb + N * 8 + x * 8);
        v[e] = {pk(p.x + q.x, p.x - q.x), pk(p.y + q.y, p.y - q.y)};
      }
    }
    __syncwarp();
    tt.forward(v, [&] {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tt.sync();
      if (tid >= 32) return;
      const bool dead = __any_sync(~0u, st.marked());
      if constexpr (kClaims) {
        load(n + G, dead ? ntiles : __shfl_sync(~0u, next, 0));
      } else if (kStager) {
        if (n + G < mine && !dead) load(n + G, blockIdx.x + (n + G) * gridDim.x);
      } else if (drain >= 0 && drain + B < mine && !dead) {
        if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
        load(drain + B, blockIdx.x + (drain + B) * gridDim.x);
      }
    });
    if (kStager && n >= SB) ok &= st.wait_on(grant + g * 8, (uint32_t)(n / G - (g < SB ? 1 : 0)) & 1u);
    const uint32_t out = kStager ? st.buf(G + n % SB) : tt.base;
#pragma unroll
    for (int i = 0; i < TT::B3; ++i) {
      const int kx = tt.q + i * TT::NT;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const Pair s = lds_pair(utw + j * 16);
        sts_pair(out + (j / BX) * (N * BX * 16) + tp_run_off<BX>(kx, j % BX), pmul_tw(v[i * J + j], s.re, s.im));
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if constexpr (kStager) {
      mbar_arrive(staged + n % SB * 8);
    } else {
      tt.sync();
      if (tid == 0) store(out, w);
      __syncwarp();
      drain = n;
    }
    set ^= 1;
  }
  if (!kStager && tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if (!ok) tp_gave_up(st, a.status);
}

// Inverse outer pass: tile order -> cubes, scaled. src and dst must not overlap. msrc: as
// k_tp_fwd's mdst.
template <int N>
__global__ void __launch_bounds__(kTpThreads<N>, 1) k_tp_inv(const __grid_constant__ CUtensorMap msrc, TpArgs a) {
  using TT = TpOuterTile<N>;
  using S = TpShape<N>;
  constexpr int J = TT::J, R = N / J, C = S::C, H = N / 2, G = S::G, B = S::B, BX = kTpBox<N>;
  extern __shared__ __align__(1024) unsigned char smraw[];
  const uint32_t sm = smem_u32(smraw);
  const TpStream<B, G> st{sm, sm + 1024, (uint32_t)kTpBuf<N>};
  const uint32_t tw = sm + 1024 + B * kTpBuf<N>, utw0 = tw + TT::kTwBytes, lin = utw0 + G * 2 * J * 16;
  const int g = threadIdx.x / TT::NT, tid = threadIdx.x % TT::NT;
  const int ntiles = a.nvol * R * H;
  constexpr bool kClaims = kTpClaims<N>;
  const int mine = kClaims ? 0 : ((int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0);
  auto load = [&](int n, int w) {  // by one thread
    if (w >= ntiles) {
      st.set_tile(n, -1);
      mbar_arrive(st.full(n));
      return;
    }
    const int vol = w / (R * H), r = w % (R * H);
    st.set_tile(n, w);
    const CUtensorMap *m = a.maps ? a.maps + vol : &msrc;
    if (a.maps) tensormap_acquire(m);
    mbar_arrive_expect_tx(st.full(n), J * N * 16);
#pragma unroll
    for (int k = 0; k < J / BX; ++k)
      tma_load_3d(st.buf(n) + k * (N * BX * 16), m, 0, ((a.maps ? 0 : vol) * (J / C) + k * BX / C) * N,
                  r * (C / BX) + k % (C / BX), st.full(n));
  };
  if (threadIdx.x == 0) {
    st.init();
    tp_grid_wait();
    for (int n = 0; n < (kClaims ? B : min(B, mine)); ++n) load(n, blockIdx.x + n * gridDim.x);
  }
  TT::fill_tw(tw, a.tw512);
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const float2 w = __ldg(a.tw512 + i * (512 / N));
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(lin + i * 8), "f"(w.x), "f"(w.y) : "memory");
  }
  tp_grid_wait();
  __syncthreads();
  TT tt(tid, 1 + g, tw);
  bool ok = true;
  int set = 0;
  for (int n = g; kClaims || n < mine; n += G) {
    int w = blockIdx.x + n * gridDim.x;
    if constexpr (kClaims) {
      // the whole group carries on or stops
      if (group_any<TT::NT>(1 + g, !st.wait(n))) {
        ok = false;
        break;
      }
      w = st.tile(n);
      if (w < 0) {  // nothing left, for the load that would follow in this buffer either
        if (tid == 0) load(n + B, ntiles);
        break;
      }
    } else {
      ok &= st.wait(n);
    }
    const int vol = w / (R * H), r = w % (R * H), y0 = r / H, zz = r % H;
    const uint32_t utw = utw0 + (g * 2 + set) * (J * 16);
    tp_step_tw<N>(utw, lin, tid, y0, zz);
    tt.at(st.buf(n));
    int next = 0;  // the tile that takes this buffer, claimed ahead of its use below
    if (kClaims && tid == 0) next = tp_claim<N>(1, n + B, gridDim.x * B, ntiles);
    Pair v[16];
#pragma unroll
    for (int i = 0; i < TT::B3; ++i)
#pragma unroll
      for (int j = 0; j < J; ++j)
        v[i * J + j] = lds_pair(tt.base + (j / BX) * (N * BX * 16) + tp_run_off<BX>(tt.q + i * TT::NT, j % BX));
    tt.sync();  // every thread has its units; the step twiddles are written
#pragma unroll
    for (int i = 0; i < TT::B3; ++i)
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const Pair s = lds_pair(utw + j * 16);
        v[i * J + j] = pmul_tw(pswap(v[i * J + j]), s.re, s.im);
      }
    tt.inverse(v, [&] {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tt.sync();
      if (tid == 0) {
        if constexpr (kClaims)
          load(n + B, st.marked() ? ntiles : next);
        else if (n + B < mine && !st.marked())
          load(n + B, blockIdx.x + (n + B) * gridDim.x);
      }
      __syncwarp();
    });
    float2 *o0 = a.dst_of(vol) + ((long long)zz * N + y0 + R * tt.row) * N, *o1 = o0 + (long long)H * N * N;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int x = tt.t + TT::R2 * e;
      const Pair p = v[e];  // swapped: re holds im
      float2 s = make_float2(lo_of(p.im) + hi_of(p.im), lo_of(p.re) + hi_of(p.re));
      float2 d = make_float2(lo_of(p.im) - hi_of(p.im), lo_of(p.re) - hi_of(p.re));
      if (a.scale != 1.0f) {
        s = make_float2(s.x * a.scale, s.y * a.scale);
        d = make_float2(d.x * a.scale, d.y * a.scale);
      }
      o0[x] = s;
      o1[x] = d;
    }
    set ^= 1;
  }
  if (!ok) tp_gave_up(st, a.status);
}

// 64 registers of a thread to and from its TMEM lane (TP_PAIR parks the filter's spectrum
// there while the signal is transformed: shared memory holds one tile only, and the
// registers hold one tile's values only).
__device__ __forceinline__ void tmem_st16(uint32_t addr, const Pair *v) {
  uint32_t r[32];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    r[4 * k] = (uint32_t)v[k].re;
    r[4 * k + 1] = (uint32_t)(v[k].re >> 32);
    r[4 * k + 2] = (uint32_t)v[k].im;
    r[4 * k + 3] = (uint32_t)(v[k].im >> 32);
  }
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t addr, Pair *v) {  // 4 units
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k].re = (f32x2)r[4 * k] | ((f32x2)r[4 * k + 1] << 32);
    v[k].im = (f32x2)r[4 * k + 2] | ((f32x2)r[4 * k + 3] << 32);
  }
}

// Middle pass over tiles of cubes in tile order. Every group reads its whole tile (and the
// filter's) before it writes the output tile, so dst may be src or, with one filter per
// cube, the filter array. With a filter a tile is two loads, the filter's and then the
// signal's, and the groups' loads alternate (load n belongs to group n % G): the filter's
// values wait in TMEM, so its buffer is free again before the signal's transform starts
// (reading a spectrum from global memory at the product took 344 us for 4 cubes of 256^3,
// this 277 otherwise alike).
template <int N, int MODE>
__global__ void __launch_bounds__(kTpThreads<N>, 1) k_tp_mid(TpArgs a) {
  using TT = TpMidTile<N>;
  using S = TpShape<N>;
  constexpr int R = TT::J, C = TT::C, H = N / 2, G = S::G, B = S::B, TILES = N * (N / R) / C;
  constexpr int LPT = MODE == TP_FWD ? 1 : 2;             // loads per tile
  constexpr long long ELEMS = (long long)R * H * C * 2;  // complex values per tile
  static_assert(TT::NT * G == kTpThreads<N> && TT::BYTES <= kTpBuf<N>, "one CTA shape for all passes");
  constexpr int kCols = MODE == TP_FWD ? 256 : 512;  // TMEM columns
  extern __shared__ __align__(1024) unsigned char smraw[];
  const uint32_t sm = smem_u32(smraw), tslot = sm + 712;
  const TpStream<B, G> st{sm, sm + 1024, (uint32_t)kTpBuf<N>};
  const uint32_t tw = sm + 1024 + B * kTpBuf<N>;
  const int g = threadIdx.x / TT::NT, tid = threadIdx.x % TT::NT;
  const int ntiles = a.nvol * TILES;
  const int mine = ((int)blockIdx.x < ntiles) ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  // Loads come in rounds of G (one per group, missing ones included so that n % G is the
  // group); tile of load n: its round's number / LPT.
  const int loads = (mine + G - 1) / G * G * LPT;
  // Tile w: cube w % nvol, tile w / nvol: the cubes' tiles against one filter run together.
  auto load = [&](int n) {  // by one thread; a missing tile's load completes at once
    const int k = (n / G / LPT) * G + n % G;  // this CTA's tile number
    if (k >= mine) {
      mbar_arrive_expect_tx(st.full(n), 0);
      return;
    }
    const int w = blockIdx.x + k * gridDim.x, vol = w % a.nvol;
    const float2 *cube = (LPT == 2 && (n / G) % 2 == 0) ? a.filt_of(vol) : a.src_of(vol);
    mbar_arrive_expect_tx(st.full(n), (uint32_t)(ELEMS * 8));
    bulk_load(st.buf(n), cube + (long long)(w / a.nvol) * ELEMS, (uint32_t)(ELEMS * 8), st.full(n));
  };
  if (threadIdx.x == 0) {
    st.init();
    tp_grid_wait();
    for (int n = 0; n < B && n < loads; ++n) load(n);
  }
  TT::fill_tw(tw, a.tw512);
  const uint32_t tmem = tp_tmem_alloc<kCols>(tslot), park = tp_tmem_warp(tmem, 1);
  tp_grid_wait();
  if (kTpClaims<N> && blockIdx.x == 0 && threadIdx.x < 2) *tp_claims<N>(threadIdx.x) = 0u;
  TT tt(tid, 1 + g, tp_tmem_warp(tmem, 0), tw);
  bool ok = true;
  int n = g;  // this group's next load
  Pair v[16];
  auto read_rows = [&] {
    tt.at(st.buf(n));
    ok &= st.wait(n);
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = lds_pair(tt.nat(tt.t + TT::R2 * e));
    __syncwarp();
  };
  auto release = [&] {  // this group is done with load n's buffer
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tt.sync();
    if (tid == 0 && n + B < loads && !st.marked()) load(n + B);
    __syncwarp();  // the TMEM instructions want the whole warp
    n += G;
  };
  // unit of output (i, j) of this thread in a spectrum's tile
  auto spec = [&](int i, int j) { return ((j * H + tt.colt + i * TT::NTC) * C + tt.c) * 2; };
  for (int k = g; k < mine; k += G) {
    const int w = blockIdx.x + k * gridDim.x, vol = w % a.nvol;
    const long long off = (long long)(w / a.nvol) * ELEMS;
    if constexpr (MODE != TP_FWD) {
      if constexpr (MODE == TP_PAIR) {
        read_rows();
        tt.forward(v, release);
      } else {
        ok &= st.wait(n);
#pragma unroll
        for (int i = 0; i < TT::B3; ++i)
#pragma unroll
          for (int j = 0; j < R; ++j) v[i * R + j] = lds_pair(st.buf(n) + spec(i, j) * 8);
        release();
      }
      tmem_st16(park, v);
      tmem_st16(park + 32, v + 8);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    read_rows();
    if constexpr (MODE == TP_FWD) {
      tt.forward(v, release);
      float2 *o = a.dst_of(vol) + off;
#pragma unroll
      for (int i = 0; i < TT::B3; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) stg_unit(o + spec(i, j), v[i * R + j]);
    } else {
      tt.forward(v, [] {});
#pragma unroll
      for (int q = 0; q < 16; q += 4) {
        Pair f[4];
        tmem_ld4(park + 4 * q, f);
#pragma unroll
        for (int m = 0; m < 4; ++m) v[q + m] = pswap(pmul(v[q + m], f[m]));
      }
      tt.inverse(v, release);
      float2 *o = a.dst_of(vol) + off;
#pragma unroll
      for (int e = 0; e < 16; ++e)
        stg_unit(o + ((tt.row * H + tt.t + TT::R2 * e) * C + tt.c) * 2, pswap(v[e]));
    }
  }
  // A group without a tile in the last round hands its buffers on all the same.
  for (; n < loads; n += G) {
    ok &= st.wait(n);
    if (tid == 0 && n + B < loads && !st.marked()) load(n + B);
  }
  if (!ok) tp_gave_up(st, a.status);
  tp_tmem_free<kCols>(tmem);
}

// A spectrum in natural order -> tile order, for calls that bring their filter's spectrum.
// Bound by the copy (16 N^3 bytes, or L2 for the small sizes; 4.7 us at N = 64, launch
// included): a block turns 32 rows (pairs of kz, C of ky) of 32 kx into 32 runs of 16 units,
// 256 bytes a run on either side. The spectrum may be what the kernel before writes, while this
// one is resident already, so it is read from L2, after the wait and not as read-only data.
template <int N>
__global__ void __launch_bounds__(256) k_tp_order(const float2 *src, float2 *dst) {
  constexpr int J = TpShape<N>::J, C = TpShape<N>::C, R = N / J, H = N / 2, KZ = 16 / C;
  __shared__ float2 rows[32][33];
  int b = blockIdx.x;
  const int x0 = b % (N / 32) * 32;
  b /= N / 32;
  const int kz0 = b % (H / KZ) * KZ;
  b /= H / KZ;
  const int k2 = b % R, g = b / R;
  const int lane = threadIdx.x & 31;
  tp_grid_wait();
  for (int i = threadIdx.x >> 5; i < 32; i += 8) {
    const int u = i >> 1, kz = 2 * (kz0 + u / C) + (i & 1), ky = g * C + u % C + J * k2;
    float2 v;
    asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];"
                 : "=f"(v.x), "=f"(v.y)
                 : "l"(src + ((long long)kz * N + ky) * N + x0 + lane)
                 : "memory");
    rows[i][lane] = v;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 512; i += 256) {
    const int x = i >> 4, u = i & 15;
    const float2 p = rows[2 * u][x], q = rows[2 * u + 1][x];
    stg_unit(dst + (((long long)g * N + x0 + x) * (R * H * C) + (k2 * H + kz0) * C + u) * 2,
             Pair{pk(p.x, q.x), pk(p.y, q.y)});
  }
}

// One convolution of a small cube in one cooperative launch: the three passes on one tile a
// CTA, grid barriers between them. Two groups per CTA, the filter's and the signal's, which
// hand over through shared memory at the product. Tiles are read and written straight from
// registers: latency is all there is (L2 round trips, exchanges, two barriers). One cube of 64^3
// 16.4 us, of 32^3 12.3, where whole planes and z tiles a block (persistent.cu) took 22.5 and
// 16.4.
template <int N>
constexpr int kTpOneThreads = 2 * TpOuterTile<N>::NT;
template <int N>
constexpr int tp_one_smem() {
  return 1024 + 2 * kTpBuf<N> + TpOuterTile<N>::kTwBytes + TpMidTile<N>::kTwBytes + TpShape<N>::J * 16 + N * 8;
}

__device__ __forceinline__ Pair ldcg_unit(const float2 *p) {
  Pair a;
  asm volatile("ld.global.cg.v2.b64 {%0, %1}, [%2];" : "=l"(a.re), "=l"(a.im) : "l"(p) : "memory");
  return a;
}

template <int N, bool REAL>
__global__ void __launch_bounds__(kTpOneThreads<N>, 1)
    k_tp_one(const float2 *sig, const float2 *filt, float2 *out, float2 *ftiles, float2 *stiles, float scale,
             const float2 *tw512, unsigned *slot, unsigned *status) {
  using OT = TpOuterTile<N>;
  using MT = TpMidTile<N>;
  constexpr int J = OT::J, R = N / J, C = MT::C, H = N / 2, NT = OT::NT, TILE = R * H * C;
  constexpr bool kTmem = MT::R2 > 1;
  static_assert(MT::NT == NT && N * J / C == R * H, "a tile of either kind per CTA and group");
  extern __shared__ __align__(1024) unsigned char smraw[];
  const uint32_t sm = smem_u32(smraw), tiles = sm + 1024, tw = tiles + 2 * kTpBuf<N>, mtw = tw + OT::kTwBytes,
                 utw = mtw + MT::kTwBytes, lin = utw + J * 16;
  const int g = threadIdx.x / NT, tid = threadIdx.x % NT, w = blockIdx.x, y0 = w / H, zz = w % H;
  const uint32_t spin = dep_wait_limit(status, kSpinLimit), buf = tiles + g * kTpBuf<N>;
  OT ot(tid, 1 + g, tw);
  ot.at(buf);
  Pair v[16];
  {
    const long long row = ((long long)zz * N + y0 + R * ot.row) * N + ot.t;
    if (REAL && g == 0) {
      const float *p = reinterpret_cast<const float *>(filt) + row, *q = p + (long long)H * N * N;
      float a[16], b[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) a[e] = __ldcg(p + OT::R2 * e), b[e] = __ldcg(q + OT::R2 * e);
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] = {pk(a[e] + b[e], a[e] - b[e]), 0ull};
    } else {
      const float2 *p = (g ? sig : filt) + row, *q = p + (long long)H * N * N;
      float2 a[16], b[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) a[e] = __ldcg(p + OT::R2 * e), b[e] = __ldcg(q + OT::R2 * e);
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] = {pk(a[e].x + b[e].x, a[e].x - b[e].x), pk(a[e].y + b[e].y, a[e].y - b[e].y)};
    }
  }
  OT::fill_tw(tw, tw512);
  MT::fill_tw(mtw, tw512);
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const float2 u = __ldg(tw512 + i * (512 / N));
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(lin + i * 8), "f"(u.x), "f"(u.y) : "memory");
  }
  uint32_t tmem = 0;
  if constexpr (kTmem) tmem = tp_tmem_alloc<64>(sm);
  __syncthreads();
  tp_step_tw<N>(utw, lin, threadIdx.x, y0, zz);
  __syncthreads();
  // unit of output (kx, j') in tile order
  auto unit = [&](int kx, int j) { return ((long long)((j / C) * N + kx) * TILE + w * C + j % C) * 2; };
  ot.forward(v, [] {});
  {
    float2 *o = g ? stiles : ftiles;
#pragma unroll
    for (int i = 0; i < OT::B3; ++i)
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const Pair s = lds_pair(utw + j * 16);
        stg_unit(o + unit(ot.q + i * NT, j), pmul_tw(v[i * J + j], s.re, s.im));
      }
  }
  bool ok = small_grid_barrier(slot, gridDim.x, status, spin);
  if (ok) {
    MT mt(tid, 1 + g, kTmem ? tp_tmem_warp(tmem, 0) : 0u, mtw);
    mt.at(buf);
    float2 *tile = (g ? stiles : ftiles) + (long long)w * TILE * 2;
    auto nat = [&](int e) { return ((mt.row * H + mt.t + MT::R2 * e) * C + mt.c) * 2; };
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = ldcg_unit(tile + nat(e));
    mt.forward(v, [] {});
    __syncthreads();
    if (g == 0) {
#pragma unroll
      for (int k = 0; k < 16; ++k) sts_pair(tiles + (k * NT + tid) * 16, v[k]);
    }
    __syncthreads();
    if (g == 1) {
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = pswap(pmul(v[k], lds_pair(tiles + (k * NT + tid) * 16)));
      mt.inverse(v, [] {});
#pragma unroll
      for (int e = 0; e < 16; ++e) stg_unit(tile + nat(e), pswap(v[e]));
    }
    ok = small_grid_barrier(slot, 2u * gridDim.x, status, spin);
  }
  small_grid_leave(slot, ok);
  if constexpr (kTmem) tp_tmem_free<64>(tmem);
  if (!ok || g == 0) return;
#pragma unroll
  for (int i = 0; i < OT::B3; ++i)
#pragma unroll
    for (int j = 0; j < J; ++j) v[i * J + j] = ldcg_unit(stiles + unit(ot.q + i * NT, j));
#pragma unroll
  for (int i = 0; i < OT::B3; ++i)
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const Pair s = lds_pair(utw + j * 16);
      v[i * J + j] = pmul_tw(pswap(v[i * J + j]), s.re, s.im);
    }
  ot.inverse(v, [] {});
  float2 *o0 = out + ((long long)zz * N + y0 + R * ot.row) * N + ot.t, *o1 = o0 + (long long)H * N * N;
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const Pair p = v[e];  // swapped: re holds im
    o0[OT::R2 * e] = make_float2((lo_of(p.im) + hi_of(p.im)) * scale, (lo_of(p.re) + hi_of(p.re)) * scale);
    o1[OT::R2 * e] = make_float2((lo_of(p.im) - hi_of(p.im)) * scale, (lo_of(p.re) - hi_of(p.re)) * scale);
  }
}

}  // namespace convgpu
