// Final-colour pass: linear float4 radiance -> packed RGBA8, the reference's
// computeFinalPixelColorsKernel (Renderer/toneMap.cu:47-71) applied to the relight output
// (indirect + direct, or indirect alone, Renderer/toneMap.cu:79-84).
//
// The per-channel encode srgb_byte(x) = floor(255.9 clamp(1.055 (x + 1e-6)^(1/2.4) - 0.055))
// is a non-decreasing step function of x with 255 steps.  The host finds each step's
// threshold once -- the smallest float whose byte reaches j, by bisection over the ordered
// bit patterns of non-negative floats, evaluating srgb_byte itself -- and the kernel maps a
// channel to the number of thresholds at or below it (an estimate, then one exact comparison in
// shared memory).
// That equals srgb_byte wherever srgb_byte is monotonic, which the oracle checks float by
// float around every threshold.  One float4 read and one 32-bit write per pixel: HBM-bound.
#include <mutex>

#include "nwprt_internal.cuh"

namespace nwprt {
namespace {

struct SrgbTable {
  float t[256];  // t[j]: smallest float with byte >= j (j >= 1); t[0] unused
};

SrgbTable build_table() {
  SrgbTable T{};
  T.t[0] = 0.f;
  for (int j = 1; j < 256; ++j) {
    uint32_t lo = 0, hi = 0x7f800000u;  // +0 .. +inf; byte(+inf) = 255
    while (lo < hi) {
      const uint32_t mid = lo + (hi - lo) / 2;
      if (srgb_byte(float_from_bits(mid)) >= (uint32_t)j) hi = mid;
      else lo = mid + 1;
    }
    T.t[j] = float_from_bits(lo);
  }
  return T;
}

const SrgbTable& table() {
  static std::once_flag once;
  static SrgbTable T;
  std::call_once(once, [] { T = build_table(); });
  return T;
}

// Number of thresholds at or below x.  The estimate g (the SFU power) is within 0.01 of the real
// step position: with x + 1e-6 >= 1e-6, lg2.approx is off by at most 3 ulp of 20, so the power by
// 2e-6 of itself and g, at most 271, by 6e-4, far below 1/2.  So the count is floor(g - 1/2) or one
// more, and one exact comparison decides.  NaN and negative x give 0, +inf gives 255.
__device__ __forceinline__ uint32_t lookup(const float* t, float x) {
  const float g = fmaf(1.055f, __powf(fmaxf(x, 0.f) + 1e-6f, 1.0f / 2.4f), -0.055f) * 255.9f;
  const int j = (int)fminf(fmaxf(g - 0.5f, 0.f), 254.f);
  return (uint32_t)j + (t[j + 1] <= x ? 1u : 0u);
}

// Pixels per thread and iteration.
constexpr int kInFlight = 3;

// HBM-bound.  A shared-memory lookup of a pseudo-random threshold meets a 3-way bank conflict, so one
// lookup per channel instead of three to four, and the table's load off the constant bank, took 16
// 1080p frames from 160 to 103 us and one 2559 x 1439 frame from 23.6 to 14.2 us.  8 blocks per SM
// (every thread slot) a whole grid apart: 64 per SM measured 18.1 us on that frame.  An ordinary load
// does not move above a store, so an iteration's loads are written before its first store: 16 frames,
// that frame and a 1080p one take 101.4 (6,540 GB/s), 13.1 and 8.5 us with three of them (two: 103.8,
// 13.4 and 8.7; four: 100.8, 13.0 and 9.1; one at a time: 119, 14.4 and 9.0).
__global__ void __launch_bounds__(256) tonemap_srgb_kernel(const __grid_constant__ SrgbTable T,
                                                           const float4* src, int64_t n, uint32_t* dst) {
  __shared__ float t[256];
  const float* table = T.t;
  asm volatile("" : "+l"(table));  // one coalesced load, not 32 constant-bank reads per warp
  t[threadIdx.x] = table[threadIdx.x];
  __syncthreads();
  let_next_start();
  stream_wait(src, dst);
  // kInFlight loads are issued before the first store, above which an ordinary load does not move
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto put = [&](int64_t at, const float4& v) {
    dst[at] = lookup(t, v.x) | (lookup(t, v.y) << 8) | (lookup(t, v.z) << 16) | (255u << 24);
  };
#pragma unroll 1
  for (; i + (kInFlight - 1) * step < n; i += kInFlight * step) {
    float4 v[kInFlight];
#pragma unroll
    for (int k = 0; k < kInFlight; ++k) v[k] = ld_stream(src + i + k * step);
#pragma unroll
    for (int k = 0; k < kInFlight; ++k) put(i + k * step, v[k]);
  }
#pragma unroll 1
  for (; i < n; i += step) put(i, ld_stream(src + i));
}

}  // namespace

void launch_tonemap_srgb(const float* src, int64_t n, uint32_t* dst, cudaStream_t st) {
  if (n < 0) fail(NWPRT_INVALID_ARG, "tonemap: negative pixel count");
  if (n == 0) return;
  if (!src || !dst) fail(NWPRT_INVALID_ARG, "tonemap: null pointer");
  if ((reinterpret_cast<uintptr_t>(src) & 15) || (reinterpret_cast<uintptr_t>(dst) & 3))
    fail(NWPRT_INVALID_ARG, "tonemap: src must be 16-byte aligned (float4), dst 4-byte aligned");
  int dev = 0, sms = 0;
  NWPRT_CUDA(cudaGetDevice(&dev));
  NWPRT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t blocks = (n + 255) / 256, cap = (int64_t)sms * 8;
  launch_overlapped(tonemap_srgb_kernel, blocks < cap ? blocks : cap, 256, 0, st, table(),
                    reinterpret_cast<const float4*>(src), n, dst);
  NWPRT_CUDA(cudaGetLastError());
}

}  // namespace nwprt
