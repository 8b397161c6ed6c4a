// SH radiance per mesh vertex and its barycentric interpolation: the SH path's shading
// (Renderer/device_functions/devicePrograms.cu:427-490) without the ray tracer.
//
// Per vertex v:  light[k] = sum_j T[v][k][j] L[j]        (RGB; j ascending, one fma per term)
//                c[v]     = | sum_k light[k] * brdf[v][k] |   (k ascending, one fma per term)
// with T the vertex's n x n transfer matrix (n = 81 at SH degree 8, 26 KB per vertex), L the
// env SH coefficients and brdf the vertex's BRDF projected on the SH basis (the reference
// projects it by sampling its material callables, devicePrograms.cu:448-474; here it is an
// input like T).  Per pixel: (1-u-v) c[i0] + u c[i1] + v c[i2].
//
// The vertex pass streams T once and does 2 n^2 FMAs per 4 n^2 bytes: HBM-bound.  One warp per
// vertex, eight per CTA: the warp copies T[v] into its shared-memory stage (bulk copies, tracked
// by an mbarrier) and brdf[v] beside it, then lane k walks rows k, k + 32, k + 64 side by side,
// each sequentially (so the sum order is the reference's), one lane per channel sums over k, and
// the other warps' copies run meanwhile.  How the rows sit in the stage:
//  * odd n: as in memory, the odd stride being free of bank conflicts.  T[v] starts 4 (v n^2 mod
//    4) bytes past a 16-byte boundary, so the stage is shifted by as much: the body moves in one
//    bulk copy, a head and a tail of at most three floats by cp.async.
//  * n a multiple of 4, T 16-byte aligned: rows an odd number of 16-byte chunks apart, read four
//    terms at a time.  One bulk copy where n / 4 is odd, else one per row.
//  * other even n, up to 8-way conflicts: as in memory all the same.  60 MB of matrices of 62: 18.5 us, 51.4 by 4-byte copies to an odd stride; of 72 (8-way) with T on no 16-byte
//    boundary 27.0 and 45.8.
//  * otherwise (multiples of 16 with T on no 16-byte boundary, and n = 2, 51.4 us against 55.4): an
//    odd stride, by 4-byte cp.async.  Matrices of 48: 37.8 us, of 80: 35.0.
// 40,000 vertices of 81 coefficients: 249 us with one row at a time (three env SH reads per term
// and row) and 16-byte cp.async, 201 with three rows side by side, 157 with bulk copies (6,930
// GB/s); 14,364 of 64: 277 us (32-way conflicts), 148 by 4-byte copies to an odd stride, 67 by
// rows; 16,146 of 25: 27.3 -> 13 us, as many CTAs per SM as fit instead of one.
#include <type_traits>

#include "nwprt_internal.cuh"

namespace nwprt {
namespace {

constexpr int kMaxN = 81;
constexpr int kWarps = 8;

enum RowForm { kOddRows, kChunkRows, kEvenRows, kSingles };  // how a matrix is staged (above)

// Shared memory in floats: the env SH (padded to 4 per coefficient), then per warp light[k] and
// brdf[v] ([kMaxN][3] each), then per warp a T staging area plus up to 3 of alignment shift,
// rounded to 16 bytes.
__host__ __device__ constexpr int stage_offset() { return (4 * kMaxN + 2 * kWarps * kMaxN * 3 + 3) & ~3; }
__host__ __device__ constexpr int row_stride(int n, RowForm form) {
  return form == kChunkRows ? ((n / 4) | 1) * 4 : form == kEvenRows ? n : n | 1;
}
__host__ __device__ constexpr int stage_stride(int n, RowForm form) { return (n * row_stride(n, form) + 3 + 3) & ~3; }

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// R = ceil(n / 32): rows per lane.  polls: limit of the wait for a matrix's bulk copy.  The call has no
// error word, so a warp whose wait runs out goes on from global memory: the results are the same.
template <int R, RowForm FORM>
__global__ void __launch_bounds__(kWarps * 32) sh_vertex_kernel(const float* __restrict__ T,
                                                                const float* __restrict__ brdf,
                                                                const float* __restrict__ L, int64_t V, int n,
                                                                float* __restrict__ out, uint32_t polls) {
  extern __shared__ __align__(16) float smem[];
  __shared__ uint64_t full[kWarps];
  const int nn = n * n, stride = row_stride(n, FORM);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float4* sL = reinterpret_cast<float4*>(smem);                         // [kMaxN] env SH
  float* light = smem + 4 * kMaxN + warp * kMaxN * 3;                   // [kMaxN][3] this warp's light[k]
  float* sb = smem + 4 * kMaxN + (kWarps + warp) * kMaxN * 3;           // [kMaxN][3] this warp's brdf[v]
  float* stage = smem + stage_offset() + warp * stage_stride(n, FORM);  // this warp's T (16-byte aligned)
  for (int i = threadIdx.x; i < n; i += blockDim.x) sL[i] = make_float4(L[i * 3], L[i * 3 + 1], L[i * 3 + 2], 0.f);
  if (threadIdx.x < kWarps) mbar_init(&full[threadIdx.x], 1);
  fence_barrier_init();
  __syncthreads();
  uint32_t parity = 0;
  int64_t v = (int64_t)blockIdx.x * kWarps + warp;
  for (; v < V; v += (int64_t)gridDim.x * kWarps) {
    const float* src = T + v * nn;
    const float* bsrc = brdf + v * n * 3;
    float* t = stage;
    if constexpr (FORM == kOddRows || FORM == kEvenRows) {
      // t[i] and src[i] share their offset modulo 16 bytes
      const int mis = (int)((reinterpret_cast<uintptr_t>(src) >> 2) & 3);
      t += mis;
      const int head = ((4 - mis) & 3) < nn ? ((4 - mis) & 3) : nn;
      const int body = (nn - head) & ~3;
      if (lane == 0) {
        // a head or tail of the matrix before, written by cp.async, may lie where this copy writes
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&full[warp], body * 4);
        if (body > 0) bulk_g2s(t + head, src + head, body * 4, &full[warp]);
      }
      if (lane < head) cp_async4(t + lane, src + lane);
      if (head + body + lane < nn) cp_async4(t + head + body + lane, src + head + body + lane);
    } else if constexpr (FORM == kChunkRows) {
      if (lane == 0) {
        mbar_arrive_expect_tx(&full[warp], nn * 4);
        if (stride == n) bulk_g2s(t, src, nn * 4, &full[warp]);
      }
      __syncwarp();  // the expected bytes are set before a row can complete
      if (stride != n)
        for (int r = lane; r < n; r += 32) bulk_g2s(t + r * stride, src + r * n, n * 4, &full[warp]);
    } else {
      for (int r = 0; r < n; ++r)
        for (int c = lane; c < n; c += 32) cp_async4(t + r * stride + c, src + r * n + c);
    }
    for (int i = lane; i < n * 3; i += 32)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(sb + i)), "l"(bsrc + i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if constexpr (FORM != kSingles) {
      if (!__all_sync(0xffffffffu, mbar_wait(&full[warp], parity, nullptr, polls))) break;
      parity ^= 1u;
    }
    __syncwarp();
    // light[k] = sum_j T[k][j] L[j], j ascending (each env SH term read once for the R rows).
    // Rows past the last repeat it.
    float l[R][3];
    const float* row[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      l[r][0] = l[r][1] = l[r][2] = 0.f;
      row[r] = t + min(lane + 32 * r, n - 1) * stride;
    }
    auto term = [&](int r, float tj, const float4& Lj) {
      l[r][0] = fmaf(tj, Lj.x, l[r][0]);
      l[r][1] = fmaf(tj, Lj.y, l[r][1]);
      l[r][2] = fmaf(tj, Lj.z, l[r][2]);
    };
    if constexpr (FORM == kChunkRows) {
      for (int j = 0; j < n; j += 4) {
        float4 q[R];
#pragma unroll
        for (int r = 0; r < R; ++r) q[r] = *reinterpret_cast<const float4*>(row[r] + j);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 Lj = sL[j + i];
#pragma unroll
          for (int r = 0; r < R; ++r) term(r, i == 0 ? q[r].x : i == 1 ? q[r].y : i == 2 ? q[r].z : q[r].w, Lj);
        }
      }
    } else {
// nines leave no rest at 9 and 81: 156.5 us for 40,000 vertices, by fours 161.5; by twelves 156.1, but
// 100,000 vertices of 9 take 41.1 us instead of 39.0
#pragma unroll 9
      for (int j = 0; j < n; ++j) {
        const float4 Lj = sL[j];
#pragma unroll
        for (int r = 0; r < R; ++r) term(r, row[r][j], Lj);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (lane + 32 * r < n) {
        float* d = light + (lane + 32 * r) * 3;
        d[0] = l[r][0];
        d[1] = l[r][1];
        d[2] = l[r][2];
      }
    __syncwarp();
    // c = | sum_k light[k] * brdf[k] |, k ascending, one lane per channel
    if (lane < 3) {
      float s = 0.f;
      for (int k = 0; k < n; ++k) s = fmaf(light[k * 3 + lane], sb[k * 3 + lane], s);
      out[v * 3 + lane] = fabsf(s);
    }
    __syncwarp();
  }
  if (FORM == kSingles || v >= V) return;
  for (; v < V; v += (int64_t)gridDim.x * kWarps) {
    for (int k = lane; k < n; k += 32) {
      float l[3] = {0.f, 0.f, 0.f};
      for (int j = 0; j < n; ++j) {
        const float tj = T[v * nn + k * n + j];
        const float4 Lj = sL[j];
        l[0] = fmaf(tj, Lj.x, l[0]);
        l[1] = fmaf(tj, Lj.y, l[1]);
        l[2] = fmaf(tj, Lj.z, l[2]);
      }
      for (int c = 0; c < 3; ++c) light[k * 3 + c] = l[c];
    }
    __syncwarp();
    if (lane < 3) {
      float s = 0.f;
      for (int k = 0; k < n; ++k) s = fmaf(light[k * 3 + lane], brdf[(v * n + k) * 3 + lane], s);
      out[v * 3 + lane] = fabsf(s);
    }
    __syncwarp();
  }
  (void)mbar_wait(&full[warp], parity, nullptr);  // the late copy ends before its memory does
}

__global__ void sh_interpolate_kernel(const float* __restrict__ vc, const int32_t* __restrict__ tri,
                                      const float* __restrict__ uv, int64_t P, int64_t V, float4* __restrict__ out,
                                      uint32_t* err) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += stride) {
    const int32_t i0 = __ldg(tri + p * 3), i1 = __ldg(tri + p * 3 + 1), i2 = __ldg(tri + p * 3 + 2);
    const float u = __ldg(uv + p * 2), w = __ldg(uv + p * 2 + 1);
    if (i0 < 0 || i1 < 0 || i2 < 0 || i0 >= V || i1 >= V || i2 >= V) {
      atomicCAS(err, 0u, (uint32_t)kDevBadIndex);
      out[p] = make_float4(0.f, 0.f, 0.f, 1.f);
      continue;
    }
    const float b0 = __fsub_rn(__fsub_rn(1.f, u), w);
    float r[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
      r[c] = fmaf(w, __ldg(vc + i2 * 3 + c), fmaf(u, __ldg(vc + i1 * 3 + c), __fmul_rn(b0, __ldg(vc + i0 * 3 + c))));
    out[p] = make_float4(r[0], r[1], r[2], 1.f);
  }
}

}  // namespace

void launch_sh_vertex(const float* T, const float* brdf, const float* L, int64_t V, int n, float* out,
                      uint32_t polls, cudaStream_t st) {
  if (V < 0 || n < 1 || n > kMaxN) fail(NWPRT_INVALID_ARG, "sh_vertex: need V >= 0 and 1 <= n <= 81");
  if (V == 0) return;
  if (!T || !brdf || !L || !out) fail(NWPRT_INVALID_ARG, "sh_vertex: null pointer");
  int dev = 0, sms = 0;
  NWPRT_CUDA(cudaGetDevice(&dev));
  NWPRT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  auto go = [&](auto kern, RowForm form) {
    const size_t smem = (size_t)(stage_offset() + kWarps * stage_stride(n, form)) * sizeof(float);
    NWPRT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;  // 1 at n = 81 (227 KB of staging), up to 8 for few coefficients
    NWPRT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kWarps * 32, smem));
    const int64_t blocks = (V + kWarps - 1) / kWarps, cap = (int64_t)sms * (per_sm > 0 ? per_sm : 1);
    kern<<<(int)(blocks < cap ? blocks : cap), kWarps * 32, smem, st>>>(T, brdf, L, V, n, out, polls);
  };
  auto rows = [&](auto form) {
    constexpr RowForm F = decltype(form)::value;
    if (n <= 32) go(sh_vertex_kernel<1, F>, F);
    else if (n <= 64) go(sh_vertex_kernel<2, F>, F);
    else go(sh_vertex_kernel<3, F>, F);
  };
  // every row of a T[v] starts on a 16-byte boundary if T does and n is a multiple of 4 (odd and even
  // rows: one form each, as an odd stride known to the compiler takes n = 81 from 16.5 to 14.5 us)
  if (n % 2) rows(std::integral_constant<RowForm, kOddRows>{});
  else if (n % 4 == 0 && (reinterpret_cast<uintptr_t>(T) & 15) == 0) rows(std::integral_constant<RowForm, kChunkRows>{});
  else if (n % 16 && n > 2) rows(std::integral_constant<RowForm, kEvenRows>{});
  else rows(std::integral_constant<RowForm, kSingles>{});
  NWPRT_CUDA(cudaGetLastError());
}

void launch_sh_interpolate(const float* vc, int64_t V, const int32_t* tri, const float* uv, int64_t P, float* out,
                           uint32_t* err, cudaStream_t st) {
  if (P < 0 || V < 0) fail(NWPRT_INVALID_ARG, "sh_interpolate: negative size");
  if (P == 0) return;
  if (!vc || !tri || !uv || !out) fail(NWPRT_INVALID_ARG, "sh_interpolate: null pointer");
  if (reinterpret_cast<uintptr_t>(out) & 15) fail(NWPRT_INVALID_ARG, "sh_interpolate: out must be 16-byte aligned");
  int dev = 0, sms = 0;
  NWPRT_CUDA(cudaGetDevice(&dev));
  NWPRT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t blocks = (P + 255) / 256, cap = (int64_t)sms * 8;
  sh_interpolate_kernel<<<(int)(blocks < cap ? blocks : cap), 256, 0, st>>>(vc, tri, uv, P, V,
                                                                             reinterpret_cast<float4*>(out), err);
  NWPRT_CUDA(cudaGetLastError());
}

}  // namespace nwprt
