// Fused x + y pass for N = 512 on pairs of values, staged through L2 as xyl2.cuh describes (the
// same items, order, ring, counters and dependencies).
//
// An item is 8 rows (X) or 8 columns (Y), 32 KB, for a team of 128 threads: 16 threads to a
// row or column of 256 units (pairs512.cuh: a radix-2 step whose halves are the lanes of a
// pair, then two radix-16 stages with one exchange, in place). A row is half a warp's own, so
// X items have no barrier before their stores are posted; Y items have two. One thread loads
// for a CTA's two teams, in the order in which it claims items: it waits for an item's
// dependencies and for one of three buffers, so a team finds its next item landed.
//
// Bound by L2 (4.3 GB through it at 512^3, half of that HBM's) and the latency of its loads:
// 560 us, where items of 2,048 values without loads ahead (k_xy_l2's form) took 675; without
// the arithmetic it takes 510. Column tiles contiguous in the ring: the same. One CTA of four
// teams and six buffers, items claimed two at a time: 580. Lag / ring 8 / 14, 10 / 18 and
// 12 / 20: 573, 567 and 574.
//
// No deadlock: a CTA's items are loaded, and so finished, in the order they were claimed, and
// an item's dependencies come earlier in the order, so the oldest unfinished item waits for
// nothing but its CTA's older items, which are done.
#pragma once

#include "pairs512.cuh"
#include "xyl2.cuh"

namespace convgpu {

struct Xy512 {
  static constexpr int N = 512, U = 256, C = XyL2Cfg<512>::C, ITEMS = N / C, TEAMS = 2, B = 3, NT = TEAMS * 128 + 32,
                       CTAS = 2;
  static constexpr int TB = C * N * 8, ROWB = U * 16;
  static constexpr int kSmem = 1024 + B * TB + 2 * U * 16;
  static_assert(C * 16 == 128, "16 threads a row or column");
};

// msrc: the source rows as (256, 2, rows), box {256, 2, C}; mscr: the ring planes, box {C, 256,
// 1}. scratch, ctr: as k_xy_l2.
template <bool INV>
__global__ void __launch_bounds__(Xy512::NT, Xy512::CTAS)
    k_xy512(const __grid_constant__ CUtensorMap msrc, const __grid_constant__ CUtensorMap mscr, float2 *scratch,
            float2 *dst, int np, float scale, const float2 *tw512, unsigned *ctr, unsigned *status) {
  using S = Xy512;
  constexpr int N = S::N, C = S::C, ITEMS = S::ITEMS, TEAMS = S::TEAMS, B = S::B;
  extern __shared__ __align__(128) unsigned char smraw[];
  const uint32_t sm = smem_u32(smraw), tw = sm + 1024 + B * S::TB, tw2 = tw + S::U * 16;
  const TpStream<B, TEAMS> st{sm, sm + 1024, (uint32_t)S::TB};  // load n is team n % TEAMS's
  // load n's buffer has been read: one of 4 barriers a team in turn, as st.full(n)
  auto freed = [&](int n) { return sm + 256 + ((n % TEAMS) * 4 + (n / TEAMS) % 4) * 8; };
  unsigned *xdone = ctr, *yread = ctr + np, *work = ctr + 2 * (long long)np;
  constexpr int ring = XyL2Cfg<512>::RING;
  const int lag = np < XyL2Cfg<512>::LAG ? np : XyL2Cfg<512>::LAG;
  const unsigned nitems = 2u * (unsigned)np * ITEMS;
  if (threadIdx.x == 0) {
    st.init();
    for (int i = 0; i < 4 * TEAMS; ++i) mbar_init(sm + 256 + i * 8, 4);
    mbar_fence_init();
  }
  for (int i = threadIdx.x; i < S::U; i += blockDim.x) {
    const float2 w = __ldg(tw512 + (i >> 4) * (i & 15) * 2), u = __ldg(tw512 + i);
    sts_pair(tw + i * 16, Pair{pk(w.x, w.x), pk(-w.y, -w.y)});
    sts_pair(tw2 + i * 16, Pair{pk(1.f, u.x), pk(0.f, -u.y)});
  }
  __syncthreads();
  const int team = (int)threadIdx.x / 128;  // TEAMS: the last warp, which loads
  auto item = [&](unsigned w, int &p, int &tl, bool &is_y) {
    long long plane;
    xyl2_item<ITEMS>((long long)w, np, lag, plane, tl, is_y);
    p = (int)plane;
  };
  if (team == TEAMS) {
    if (threadIdx.x & 31) return;
    const uint32_t spin = dep_wait_limit(status, kXyL2Spin);
    bool landed = true, met = true;
    unsigned next = atomicAdd(work, 1u);
    for (int n = 0, none = 0; none < TEAMS; ++n) {
      const unsigned w = next;
      if (w >= nitems) {  // nothing left: says so to each team
        st.set_tile(n, -1);
        mbar_arrive(st.full(n));
        ++none;
        continue;
      }
      int p, tl;
      bool is_y;
      item(w, p, tl, is_y);
      next = atomicAdd(work, 1u);
      const unsigned *dep = is_y ? xdone + p : (p >= ring ? yread + (p - ring) : nullptr);
      // once one has given up none waits any more
      if (dep && !wait_count(dep, ITEMS, met ? spin : 0u)) met = false;
      if (n >= B) {
        const uint32_t bar = freed(n - B), parity = (uint32_t)((n - B) / (4 * TEAMS)) & 1u;
        bool ok = mbar_try_wait(bar, parity);
        if (!ok && !st.marked()) {
          ok = mbar_wait_bounded(bar, parity);
          if (!ok) asm volatile("st.shared.u32 [%0], %1;" ::"r"(st.mark()), "r"(1u) : "memory");
        }
        landed &= ok;
      }
      st.set_tile(n, (int)w);
      if (st.marked()) {
        mbar_arrive(st.full(n));
        continue;
      }
      mbar_arrive_expect_tx(st.full(n), S::TB);
      if (is_y) {
        asm volatile("fence.proxy.async.global;" ::: "memory");  // generic stores -> TMA reads
        tma_load_3d(st.buf(n), &mscr, tl * C, 0, p % ring, st.full(n));
        tma_load_3d(st.buf(n) + S::TB / 2, &mscr, tl * C, 256, p % ring, st.full(n));
      } else {
        tma_load_3d(st.buf(n), &msrc, 0, 0, p * N + tl * C, st.full(n));
      }
    }
    if (!met && status) atomicOr(status, kStatusQueueWait);
    if (!landed) tp_gave_up(st, status);
    return;
  }
  const int tid = threadIdx.x % 128;
  auto barrier = [&] { group_sync<128>(1 + team); };
  // Every item's first barrier, whatever the item is, also says whether a warp's wait has given
  // up, so that the whole team carries on or stops (a barrier of its own for that: 35 us more).
  bool ok = true;
  auto stopped = [&](bool here) {
    const bool stop = group_any<128>(1 + team, here);
    ok &= !stop;
    return stop;
  };
  Pair v[16];
  for (int n = team;; n += TEAMS) {
    const bool got = st.wait(n);
    const int w = got ? st.tile(n) : -1;
    if (w < 0) {
      stopped(!got);
      break;
    }
    int p, tl;
    bool is_y;
    item((unsigned)w, p, tl, is_y);
    const uint32_t buf = st.buf(n);
    // This warp has read the buffer for the last time.
    auto release = [&] {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (tid % 32 == 0) mbar_arrive(freed(n));
      __syncwarp();
    };
    if (is_y) {
      if (tid == 0) red_relaxed_add_u32(yread + p, 1u);  // landed: the slot may be rewritten
      __syncwarp();
      const int c = tid % C, t = tid / C;
      const UnitColumn<C * 16> col{buf + (uint32_t)c * 16, tw, tw2, t};
      col.load(v, buf + (uint32_t)c * 8, C * 8, 1.f);
      if (INV) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = pswap(v[e]);
      }
      col.stage1(v);
      if (stopped(false)) break;
      col.write1(v);
      barrier();
      col.read2(v);
      release();
      PDft<16>::run(v);
      float2 *o = dst + (long long)p * N * N + tl * C + c + (long long)2 * t * N;
#pragma unroll
      for (int k = 0; k < 16; ++k) {  // rows 2 (t + 16 k) and the next
        const Pair r = INV ? pswap(v[k]) : v[k];
        o[32ll * k * N] = make_float2(lo_of(r.re) * scale, lo_of(r.im) * scale);
        o[32ll * k * N + N] = make_float2(hi_of(r.re) * scale, hi_of(r.im) * scale);
      }
    } else {
      const int row = tid / 16, t = tid % 16;
      const uint32_t mine = buf + (uint32_t)row * S::ROWB;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float2 a = lds_f2(mine + (t + 16 * e) * 8), b = lds_f2(mine + (t + 16 * e + 256) * 8);
        v[e] = {pk(a.x + b.x, a.x - b.x), pk(a.y + b.y, a.y - b.y)};
        if (INV) v[e] = pswap(v[e]);
      }
      const UnitColumn<16> r{mine, tw, tw2, t};
      r.stage1(v);
      __syncwarp();
      // slot of (k1, t): 16 k1 + (t ^ k1), all banks for either side
#pragma unroll
      for (int k = 0; k < 16; ++k) sts_pair(mine + (16 * k + (t ^ k)) * 16, v[k]);
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = lds_pair(mine + (16 * t + (k ^ t)) * 16);
      release();
      PDft<16>::run(v);
      float2 *o = scratch + (long long)(p % ring) * N * N + (long long)(tl * C + row) * N + 2 * t;
#pragma unroll
      for (int k = 0; k < 16; ++k) {  // columns 2 (t + 16 k) and the next
        const Pair u = INV ? pswap(v[k]) : v[k];
        stg_unit(o + 32 * k, Pair{pk(lo_of(u.re), lo_of(u.im)), pk(hi_of(u.re), hi_of(u.im))});
      }
      if (stopped(false)) break;  // every thread's stores issued; orders them before the release
      if (tid == 0) red_release_add_u32(xdone + p, 1u);
      __syncwarp();
    }
  }
  if (!ok) tp_gave_up(st, status);
}

}  // namespace convgpu
