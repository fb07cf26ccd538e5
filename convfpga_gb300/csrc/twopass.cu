// Launchers of the two-pass 3D transform (twopass.cuh) for N = 32 to 256, and its scratch
// cubes. One persistent CTA per SM; launches read their operands through plain pointers, and
// only the runs of tile order go through a tensor map.
#define CONVGPU_PASS_LAUNCH_IMPL
#include "engine_internal.h"
#include "pass_launch.cuh"
#include "twopass.cuh"

#include <algorithm>
#include <type_traits>

namespace convgpu {

bool tp_size(int n) { return n == 32 || n == 64 || n == 128 || n == 256; }

namespace {

template <class K, class... M>
cudaError_t launch_blocks(K kern, int smem, int threads, long long blocks, cudaStream_t s, const M &...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e != cudaSuccess) cudaGetLastError();  // reported here, not by the next launch's check
  return e;
}

// Persistent: one CTA per SM at most.
template <class K, class... M>
cudaError_t launch(K kern, int &done, int smem, int threads, long long tiles, cudaStream_t s, const M &...args) {
  if (tiles <= 0 || tiles > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  const cudaError_t e = set_smem_once(kern, smem, done);
  if (e != cudaSuccess) return e;
  return launch_blocks(kern, smem, threads, std::min<long long>(tiles, sm_count()), s, args...);
}

template <int N>
bool encode_tiles(CUtensorMap *m, const void *cubes, int nvol) {
  using S = TpShape<N>;
  return encode_runs_map(m, cubes, 2 * kTpBox<N>, (long long)nvol * N * S::J / S::C,
                         (N / S::J) * (N / 2) * (S::C / kTpBox<N>), N);
}

template <int N>
cudaError_t fwd(const TpArgs &a, bool real, const CUtensorMap &m, const CUtensorMap &m2, cudaStream_t s) {
  const long long tiles = (long long)a.nvol * (N / TpShape<N>::J) * (N / 2);
  static int done[2] = {0, 0};
  constexpr int smem = tp_outer_smem<N>(), threads = kTpFwdThreads<N>;
  return real ? launch(k_tp_fwd<N, true>, done[1], smem, threads, tiles, s, m, m2, a)
              : launch(k_tp_fwd<N, false>, done[0], smem, threads, tiles, s, m, m2, a);
}

template <int N>
cudaError_t inv(const TpArgs &a, const CUtensorMap &m, cudaStream_t s) {
  const long long tiles = (long long)a.nvol * (N / TpShape<N>::J) * (N / 2);
  static int done = 0;
  return launch(k_tp_inv<N>, done, tp_outer_smem<N>(), kTpThreads<N>, tiles, s, m, a);
}

template <int N>
cudaError_t mid(const TpArgs &a, int mode, cudaStream_t s) {
  const long long tiles = (long long)a.nvol * N * TpShape<N>::J / TpShape<N>::C;
  static int done[3] = {0, 0, 0};
  constexpr int smem = tp_mid_smem<N>(), threads = kTpThreads<N>;
  switch (mode) {
    case TP_PAIR: return launch(k_tp_mid<N, TP_PAIR>, done[0], smem, threads, tiles, s, a);
    case TP_SPECTRUM: return launch(k_tp_mid<N, TP_SPECTRUM>, done[1], smem, threads, tiles, s, a);
    case TP_FWD: return launch(k_tp_mid<N, TP_FWD>, done[2], smem, threads, tiles, s, a);
    default: return cudaErrorInvalidValue;
  }
}

template <int N>
cudaError_t order(const float2 *src, float2 *dst, cudaStream_t s) {
  return launch_blocks(k_tp_order<N>, 0, 256, (long long)N * N * N / 1024, s, src, dst);
}

TpArgs args(int n, const void *src, void *dst, int nvol, const float2 *tw512) {
  TpArgs a{};
  a.src = static_cast<const float2 *>(src);
  a.dst = static_cast<float2 *>(dst);
  a.src_vol = a.dst_vol = (long long)n * n * n;
  a.nvol = nvol;
  a.scale = 1.f;
  a.tw512 = tw512;
  a.status = device_status_address();
  return a;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// N = 32, 64, 128, 256. One that could not be allocated is not asked for again, call by call,
// before release_tp.
struct TpScratch {
  float2 *p = nullptr;
  bool none = false;      // not to be had, or given back
  bool captured = false;  // a graph may hold it
} g_scratch[4];

// Calls f with N as a compile-time constant.
template <class F>
cudaError_t with_size(int n, F &&f) {
  switch (n) {
    case 32: return f(std::integral_constant<int, 32>{});
    case 64: return f(std::integral_constant<int, 64>{});
    case 128: return f(std::integral_constant<int, 128>{});
    case 256: return f(std::integral_constant<int, 256>{});
    default: return cudaErrorNotSupported;
  }
}

}  // namespace

int tp_scratch_cubes(int n) {
  return n == 32 ? kTpScratchCubes32
                 : (n == 64 ? kTpScratchCubes64 : (n == 128 ? kTpScratchCubes128 : kTpScratchCubes256));
}

float2 *tp_scratch(int n, bool may_allocate) {
  TpScratch &t = g_scratch[n == 32 ? 0 : (n == 64 ? 1 : (n == 128 ? 2 : 3))];
  if (!t.p && !t.none && may_allocate) {
    void *q = nullptr;
    if (!allocation_fails_on_purpose() &&
        cudaMalloc(&q, (size_t)tp_scratch_cubes(n) * n * n * n * sizeof(float2)) == cudaSuccess) {
      t.p = static_cast<float2 *>(q);
    } else {
      cudaGetLastError();
      t.none = true;
    }
  }
  t.captured |= t.p && !may_allocate;
  return t.p;
}

bool give_back_tp() {
  bool any = false;
  for (auto &t : g_scratch) {
    if (!t.p || t.captured) continue;
    if (!any) cudaDeviceSynchronize();
    any = true;
    cudaFree(t.p);
    t.p = nullptr;
    t.none = true;
  }
  return any;
}

void release_tp() {
  for (auto &t : g_scratch) {
    if (t.p) cudaFree(t.p);
    t = TpScratch{};
  }
}

bool tp_encode_tiles(CUtensorMap *m, const void *cubes, int n, int nvol) {
  return with_size(n, [&](auto k) {
           return encode_tiles<decltype(k)::value>(m, cubes, nvol) ? cudaSuccess : cudaErrorNotSupported;
         }) == cudaSuccess;
}

cudaError_t launch_tp_fwd(int n, const void *src, float2 *dst, int nvol, bool real, const float2 *tw512,
                          cudaStream_t s, const float2 *src2, float2 *dst2, int nvol2) {
  TpArgs a = args(n, src, dst, nvol + nvol2, tw512);
  a.first = nvol;
  a.src2 = src2;
  CUtensorMap m, m2;
  if (!tp_size(n) || !aligned16(src) || !aligned16(src2) || !tp_encode_tiles(&m, dst, n, nvol) ||
      !tp_encode_tiles(&m2, nvol2 ? dst2 : dst, n, nvol2 ? nvol2 : nvol))
    return cudaErrorNotSupported;
  return with_size(n, [&](auto k) { return fwd<decltype(k)::value>(a, real, m, m2, s); });
}

cudaError_t launch_tp_inv(int n, const float2 *src, float2 *dst, int nvol, float scale, const float2 *tw512,
                          cudaStream_t s) {
  TpArgs a = args(n, src, dst, nvol, tw512);
  a.scale = scale;
  CUtensorMap m;
  if (!tp_size(n) || !tp_encode_tiles(&m, src, n, nvol)) return cudaErrorNotSupported;
  return with_size(n, [&](auto k) { return inv<decltype(k)::value>(a, m, s); });
}

cudaError_t launch_tp_mid(int n, int mode, const float2 *src, float2 *dst, const float2 *filt, long long filt_vol,
                          int nvol, const float2 *tw512, cudaStream_t s) {
  TpArgs a = args(n, src, dst, nvol, tw512);
  a.filt = filt;
  a.filt_vol = filt_vol;
  if (!tp_size(n) || !aligned16(src) || !aligned16(dst) || (mode != TP_FWD && !aligned16(filt)))
    return cudaErrorNotSupported;
  return with_size(n, [&](auto k) { return mid<decltype(k)::value>(a, mode, s); });
}

cudaError_t launch_tp_order(int n, const float2 *src, float2 *dst, cudaStream_t s) {
  return with_size(n, [&](auto k) { return order<decltype(k)::value>(src, dst, s); });
}

cudaError_t launch_tp_one(int n, const float2 *sig, const float2 *filt, float2 *out, float2 *ftiles, float2 *stiles,
                          float scale, bool real, const float2 *tw512, unsigned *slot, unsigned *status,
                          cudaStream_t s) {
  void *a[] = {&sig, &filt, &out, &ftiles, &stiles, &scale, &tw512, &slot, &status};
  auto go = [&](auto k) {
    constexpr int N = decltype(k)::value;
    static_assert(tp_one_smem<N>() <= 48 << 10, "no attribute needed");
    const void *kern = real ? (const void *)k_tp_one<N, true> : (const void *)k_tp_one<N, false>;
    return cudaLaunchCooperativeKernel(kern, dim3(N / TpShape<N>::J * (N / 2)), dim3(kTpOneThreads<N>), a,
                                       tp_one_smem<N>(), s);
  };
  if (sm_count() < 128) return cudaErrorNotSupported;  // every CTA resident, one a SM
  if (n == 32) return go(std::integral_constant<int, 32>{});
  if (n == 64) return go(std::integral_constant<int, 64>{});
  return cudaErrorNotSupported;
}

cudaError_t launch_tp_fwd_table(int n, const float2 *const *srcs, const CUtensorMap *dst_maps, int nvol,
                                const float2 *tw512, cudaStream_t s) {
  TpArgs a = args(n, nullptr, nullptr, nvol, tw512);
  a.srcs = srcs;
  a.maps = dst_maps;
  CUtensorMap m{};
  return with_size(n, [&](auto k) { return fwd<decltype(k)::value>(a, false, m, m, s); });
}

cudaError_t launch_tp_inv_table(int n, const CUtensorMap *src_maps, float2 *const *dsts, int nvol, float scale,
                                const float2 *tw512, cudaStream_t s) {
  TpArgs a = args(n, nullptr, nullptr, nvol, tw512);
  a.scale = scale;
  a.maps = src_maps;
  a.dsts = dsts;
  CUtensorMap m{};
  return with_size(n, [&](auto k) { return inv<decltype(k)::value>(a, m, s); });
}

cudaError_t launch_tp_mid_table(int n, const float2 *const *srcs, float2 *const *dsts, const float2 *const *filts,
                                int nvol, const float2 *tw512, cudaStream_t s) {
  TpArgs a = args(n, nullptr, nullptr, nvol, tw512);
  a.srcs = srcs;
  a.dsts = dsts;
  a.filts = filts;
  return with_size(n, [&](auto k) { return mid<decltype(k)::value>(a, TP_PAIR, s); });
}

template <int N>
static cudaError_t prepare() {
  cudaError_t e = cudaSuccess;
  const int outer = tp_outer_smem<N>(), middle = tp_mid_smem<N>();
  auto set = [&](auto kern, int smem) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  };
  set(k_tp_fwd<N, false>, outer);
  set(k_tp_inv<N>, outer);
  set(k_tp_mid<N, TP_PAIR>, middle);
  return e;
}

cudaError_t prepare_tp(int n) {
  return with_size(n, [](auto k) { return prepare<decltype(k)::value>(); });
}

}  // namespace convgpu
