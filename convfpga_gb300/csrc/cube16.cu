// Convolutions of 16^3 cubes, one CTA per cube and one launch per batch: a cube is 32 KB, so
// both transforms, the product and the inverse stay in registers and one shared-memory
// buffer, and a batch of any size is read and written once.
//
// A thread holds 16 values along one axis, a whole transform of that axis: no twiddles. The
// signal and its filter are the two lanes of packed pairs (tilefft.cuh), so their forward
// transforms are one, also under a shared filter (32 KB from L2 for every cube, cheaper than
// a launch of its own), and the product needs no other operand. Forward z, y, x; product;
// inverse x, y, z: z to y and back exchange across the CTA, y to x inside a half warp.
//
// What bounds it: for one cube the latency of a load, six 16-point transforms and four
// exchanges after one launch (the cooperative launch with two grid barriers took 10.7 us);
// for a batch the separate axis passes moved every cube seven times through L2 in seven
// launches. The reference runs one FFT size per bitstream and one cube at a time
// (kernels/common/conv_config.h.in:8-11).
#include <algorithm>

#include "engine_internal.h"
#include "tilefft.cuh"

namespace convgpu {
namespace {

enum FilterKind : int { kComplex = 0, kReal = 1, kSpectrum = 2 };

struct Cube16Args {
  const float2 *sig;
  const float2 *filt;  // kReal: 4096 floats per filter
  float2 *out;
  long long filt_vol;  // filter values between cubes (0: one for all)
  float scale;
  const float2 *const *sigs;  // jobs at unrelated addresses, else null
  const float2 *const *filts;
  float2 *const *outs;
};

constexpr int kThreads = 256, kSmem = 4096 * 16;

// Unit (z, y, x) of the exchange buffer, x swizzled by y so that 8 lanes along x or along y
// cover all banks.
__device__ __forceinline__ uint32_t unit(int z, int y, int x) { return (uint32_t)(z * 256 + y * 16 + (x ^ (y & 7))) * 16; }

template <int KIND>
__global__ void __launch_bounds__(kThreads, 2) k_cube16(Cube16Args a) {
  extern __shared__ __align__(128) unsigned char smraw[];
  const uint32_t sm = smem_u32(smraw);
  const int tid = threadIdx.x, hi = tid >> 4, lo = tid & 15;
  const long long cube = blockIdx.x;
  const float2 *sig = a.sigs ? a.sigs[cube] : a.sig + cube * 4096;
  const float2 *filt = a.filts ? a.filts[cube] : a.filt + (KIND == kReal ? 0 : cube * a.filt_vol);
  float2 *out = a.outs ? a.outs[cube] : a.out + cube * 4096;
  Pair v[16];
  {  // column (y, x) = tid along z
    float2 s[16], f[16];
#pragma unroll
    for (int z = 0; z < 16; ++z) s[z] = sig[z * 256 + tid];
#pragma unroll
    for (int z = 0; z < 16; ++z) {
      if constexpr (KIND == kComplex)
        f[z] = filt[z * 256 + tid];
      else if constexpr (KIND == kReal)
        f[z] = make_float2(reinterpret_cast<const float *>(filt)[cube * a.filt_vol + z * 256 + tid], 0.f);
      else
        f[z] = make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int z = 0; z < 16; ++z) v[z] = {pk(s[z].x, f[z].x), pk(s[z].y, f[z].y)};
  }
  PDft<16>::run(v);
#pragma unroll
  for (int z = 0; z < 16; ++z) sts_pair(sm + unit(z, hi, lo), v[z]);
  __syncthreads();
  // row (z, x) = (hi, lo) along y: this thread's own slots from here to the inverse z pass
#pragma unroll
  for (int y = 0; y < 16; ++y) v[y] = lds_pair(sm + unit(hi, y, lo));
  PDft<16>::run(v);
#pragma unroll
  for (int y = 0; y < 16; ++y) sts_pair(sm + unit(hi, y, lo), v[y]);
  __syncwarp();
  // row (z, y) = (hi, lo) along x
#pragma unroll
  for (int x = 0; x < 16; ++x) v[x] = lds_pair(sm + unit(hi, lo, x));
  PDft<16>::run(v);
#pragma unroll
  for (int x = 0; x < 16; ++x) {
    const float2 s = make_float2(lo_of(v[x].re), lo_of(v[x].im));
    const float2 f = KIND == kSpectrum ? filt[tid * 16 + x] : make_float2(hi_of(v[x].re), hi_of(v[x].im));
    // swapped (im, re): the inverse is a forward transform of it; the other lane is free
    v[x] = {pk(s.x * f.y + s.y * f.x, 0.f), pk(s.x * f.x - s.y * f.y, 0.f)};
  }
  PDft<16>::run(v);
  __syncwarp();
#pragma unroll
  for (int x = 0; x < 16; ++x) sts_pair(sm + unit(hi, lo, x), v[x]);
  __syncwarp();
#pragma unroll
  for (int y = 0; y < 16; ++y) v[y] = lds_pair(sm + unit(hi, y, lo));
  PDft<16>::run(v);
#pragma unroll
  for (int y = 0; y < 16; ++y) sts_pair(sm + unit(hi, y, lo), v[y]);
  __syncthreads();
#pragma unroll
  for (int z = 0; z < 16; ++z) v[z] = lds_pair(sm + unit(z, hi, lo));
  PDft<16>::run(v);
#pragma unroll
  for (int z = 0; z < 16; ++z) out[z * 256 + tid] = make_float2(lo_of(v[z].im) * a.scale, lo_of(v[z].re) * a.scale);
}

// Forward transforms of 16^3 cubes, two to a CTA, one in each lane (dst may be src): one launch
// instead of one per axis: 1 to 300 cubes 6.2 us instead of 12.3 to 20.5, 1000 cubes 14.4
// instead of 41.8.
__global__ void __launch_bounds__(kThreads, 2) k_spectrum16(const float2 *src, float2 *dst, int cubes) {
  extern __shared__ __align__(128) unsigned char smraw[];
  const uint32_t sm = smem_u32(smraw);
  const int tid = threadIdx.x, hi = tid >> 4, lo = tid & 15;
  const long long at = (long long)blockIdx.x * 8192 + tid;
  const bool two = 2 * (int)blockIdx.x + 1 < cubes;
  Pair v[16];
  {
    float2 a[16], b[16];
#pragma unroll
    for (int z = 0; z < 16; ++z) a[z] = src[at + z * 256];
#pragma unroll
    for (int z = 0; z < 16; ++z) b[z] = two ? src[at + 4096 + z * 256] : make_float2(0.f, 0.f);
#pragma unroll
    for (int z = 0; z < 16; ++z) v[z] = {pk(a[z].x, b[z].x), pk(a[z].y, b[z].y)};
  }
  PDft<16>::run(v);
#pragma unroll
  for (int z = 0; z < 16; ++z) sts_pair(sm + unit(z, hi, lo), v[z]);
  __syncthreads();
#pragma unroll
  for (int y = 0; y < 16; ++y) v[y] = lds_pair(sm + unit(hi, y, lo));
  PDft<16>::run(v);
#pragma unroll
  for (int y = 0; y < 16; ++y) sts_pair(sm + unit(hi, y, lo), v[y]);
  __syncwarp();
#pragma unroll
  for (int x = 0; x < 16; ++x) v[x] = lds_pair(sm + unit(hi, lo, x));
  PDft<16>::run(v);
  __syncwarp();
#pragma unroll
  for (int x = 0; x < 16; ++x) sts_pair(sm + unit(hi, lo, x), v[x]);
  __syncthreads();
#pragma unroll
  for (int z = 0; z < 16; ++z) {
    const Pair p = lds_pair(sm + unit(z, hi, lo));
    dst[at + z * 256] = make_float2(lo_of(p.re), lo_of(p.im));
    if (two) dst[at + 4096 + z * 256] = make_float2(hi_of(p.re), hi_of(p.im));
  }
}

cudaError_t launch(int kind, const Cube16Args &a, int cubes, cudaStream_t s) {
  static int done[3][64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorNotSupported;
  auto kern = kind == kReal ? k_cube16<kReal> : (kind == kSpectrum ? k_cube16<kSpectrum> : k_cube16<kComplex>);
  if (!done[kind][dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return e;
    done[kind][dev] = 1;
  }
  kern<<<cubes, kThreads, kSmem, s>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_cube16(const float2 *sig, const void *filt, float2 *out, int cubes, bool per_signal, bool real,
                          bool spectrum, float scale, cudaStream_t s) {
  Cube16Args a{};
  a.sig = sig;
  a.filt = static_cast<const float2 *>(filt);
  a.out = out;
  a.filt_vol = per_signal ? 4096 : 0;
  a.scale = scale;
  return launch(spectrum ? kSpectrum : (real ? kReal : kComplex), a, cubes, s);
}

cudaError_t launch_spectrum16(const float2 *src, float2 *dst, int cubes, cudaStream_t s) {
  static int done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorNotSupported;
  if (!done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(k_spectrum16, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return e;
    done[dev] = 1;
  }
  k_spectrum16<<<cubes / 2 + cubes % 2, kThreads, kSmem, s>>>(src, dst, cubes);
  return cudaGetLastError();
}

cudaError_t launch_cube16_table(const float2 *const *sigs, const float2 *const *filts, float2 *const *outs, int cubes,
                                float scale, cudaStream_t s) {
  Cube16Args a{};
  a.sigs = sigs;
  a.filts = filts;
  a.outs = outs;
  a.scale = scale;
  return launch(kComplex, a, cubes, s);
}

cudaError_t prepare_cube16() {
  return cudaFuncSetAttribute(k_cube16<kComplex>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
}

}  // namespace convgpu
