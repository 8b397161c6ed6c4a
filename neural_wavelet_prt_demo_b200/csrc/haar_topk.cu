// Cubemap Haar transform + top-K wavelet selection: one thread-block cluster per env map for
// single maps and small batches, one persistent CTA per map for large batches
// (haar_topk_batch_kernel, described where it is defined).
//
// The reference only loads precomputed results (waveletcoeffs/<name>.npy and
// waveletstrength/<name>.npy, Renderer/EnvironmentMap.cpp:97-108); the transform and
// the selection order are defined by the oracle (oracle/nwprt_oracle.c:
// orc_haar_face / orc_haar_topk) and reproduced here bit for bit:
//  * per face, non-standard 2-D Haar with orthonormal 1/2 factors, Mallat layout,
//    evaluated with the same FP32 adds/multiplies (no contraction: __fadd_rn etc.);
//  * key = |0.212671 r + 0.715160 g + 0.072169 b| (EnvironmentMap.cpp:149-151), NaN -> 0;
//  * order = key descending, flat index face*S*S + row*S + col ascending.
//
// Cluster form: 6 CTAs (one per face) of 256 threads.  Nothing but the inputs and outputs
// touches global memory, and the face never goes through shared memory:
//  * Haar in registers.  Thread t owns the 4x4 texel block at block coordinates
//    (bi, bj) = Morton(t) (bj on the even bits) and evaluates the first two levels on it
//    alone: 15 detail coefficients stay in its registers, one LL value moves on.  Because
//    the LL grid is held in Morton order, every 2x2 block of the next level sits in 4
//    consecutive lanes and the next 16 in one warp, so two more levels are warp shuffles.
//    The (at most 16) LL values left go through shared memory to warp 0, which finishes
//    the last levels the same way: one block barrier for the whole transform.  The
//    coefficients of those upper levels fill exactly the top-left (S/4)^2 block of the
//    face, one per thread, so each thread owns 16 coefficients.
//  * The bin of the K-th largest key, in a window of 16 binades below the map's largest key at
//    1/16 binade: each CTA histograms its keys (registers -> shared atomics), and every CTA sums
//    the six histograms through distributed shared memory.  Two cluster barriers (the maximum,
//    the histograms), where a radix select over the keys took one per pass of four.
//  * The keys of that bin and above are listed in all six CTAs, bin by bin, and each CTA ranks its
//    own face's among their bin's (a few dozen) and writes those of rank below K: one barrier.
//  * Maps whose window holds fewer than K keys, or more than 512 too many in the last bin (ties),
//    take a 4-pass 8-bit radix select; ties at the threshold are then ranked by flat index with a
//    per-face bitmap and popcount prefixes, and every CTA ranks a sixth of the winners.
// One 6 x 64 x 64 map, graph launches: K = 64 10.6 -> 5.7 us, K = 300 14.2 -> 6.8, K = 1024
// 25.0 -> 9.8 (radix select for all maps, all-pairs ranking, before).
#include <cooperative_groups.h>

#include <type_traits>

#include "nwprt_internal.cuh"

namespace cg = cooperative_groups;

namespace nwprt {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxS = 64;
constexpr int kMaxK = 1024;

struct Winner {
  float r, g, b;
  int32_t idx;
};

// Coefficients the cluster form lists and ranks directly: the K winners and up to 512 more that
// share the last one's bin.
__host__ __device__ constexpr int list_cap(int K) { return K + 512; }

struct HaarSmem {
  uint32_t* hist;    // [2][256] this face's histogram: of the window; general form: of a pass (double buffered)
  uint32_t* seg;     // [256] a window bin's part of the list: start | length << 16
  uint32_t* cur;     // [256] where this face's next key of the bin goes
  uint32_t* kmax;    // [6 * kWarps] every warp's largest key
  float* upper;      // [(S/4)^2][3] coefficients of the top-left (S/4)^2 block
  float* llg;        // [16][3] LL values handed to warp 0 for the last levels
  uint32_t* bits;    // [S*S/32] ties at the threshold, by flat index within the face
  uint32_t* wpre;    // [S*S/32] exclusive popcount prefix of `bits`
  uint64_t* gkey;    // [list_cap(K)] composite keys of the listed coefficients (in every CTA)
  Winner* gval;      // [list_cap(K)] the values of this face's; general form: of all K winners
  int* warp_tot;     // [kWarps]
  int* scal;         // scalars
};

// scal[] slots
constexpr int kScPrefix = 0, kScMask = 1, kScRemaining = 2, kScCounter = 3, kScEq = 8;  // eq: [6]
constexpr int kScListed = 14;                // cluster form: keys listed
constexpr int kScNAbove = 16;                // batched kernel: keys in the final list
constexpr int kScLevels = 17;                // batched kernel: winners written so far, those of level 2 apart: [2]
constexpr int kScLeast = 19, kScMost = 20;   // batched kernel: of the keys marked
constexpr int kScTied = 21;                  // batched kernel: the keys marked are all equal

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

__host__ __device__ inline size_t smem_layout(int S, int K, char* base, HaarSmem* L) {
  const int G = S < 4 ? 1 : S / 4;
  const int nw = (S * S + 31) / 32;
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o = align16(o + bytes); return at; };
  size_t oH = take(sizeof(uint32_t) * 512);
  size_t oS2 = take(sizeof(uint32_t) * 256);
  size_t oC2 = take(sizeof(uint32_t) * 256);
  size_t oM = take(sizeof(uint32_t) * 6 * kWarps);
  size_t oU = take(sizeof(float) * 3 * G * G);
  size_t oL = take(sizeof(float) * 3 * 16);
  size_t oB = take(sizeof(uint32_t) * nw);
  size_t oP = take(sizeof(uint32_t) * nw);
  size_t oG = take(sizeof(uint64_t) * list_cap(K));
  size_t oV = take(sizeof(Winner) * list_cap(K));
  size_t oW = take(sizeof(int) * kWarps);
  size_t oS = take(sizeof(int) * 32);
  if (L) {
    L->hist = (uint32_t*)(base + oH);
    L->seg = (uint32_t*)(base + oS2);
    L->cur = (uint32_t*)(base + oC2);
    L->kmax = (uint32_t*)(base + oM);
    L->upper = (float*)(base + oU);
    L->llg = (float*)(base + oL);
    L->bits = (uint32_t*)(base + oB);
    L->wpre = (uint32_t*)(base + oP);
    L->gkey = (uint64_t*)(base + oG);
    L->gval = (Winner*)(base + oV);
    L->warp_tot = (int*)(base + oW);
    L->scal = (int*)(base + oS);
  }
  return o;
}

__device__ __forceinline__ void haar4(float a, float b, float c, float d, float& ll, float& hl,
                                      float& lh, float& hh) {
  const float s0 = __fadd_rn(a, b), d0 = __fsub_rn(a, b);
  const float s1 = __fadd_rn(c, d), d1 = __fsub_rn(c, d);
  ll = __fmul_rn(__fadd_rn(s0, s1), 0.5f);
  hl = __fmul_rn(__fadd_rn(d0, d1), 0.5f);
  lh = __fmul_rn(__fsub_rn(s0, s1), 0.5f);
  hh = __fmul_rn(__fsub_rn(d0, d1), 0.5f);
}

__device__ __forceinline__ uint32_t wavelet_key_bits(float r, float g, float b) {
  float t = __fmul_rn(0.212671f, r);
  t = __fadd_rn(t, __fmul_rn(0.715160f, g));
  t = __fadd_rn(t, __fmul_rn(0.072169f, b));
  return __float_as_uint(fmaxf(fabsf(t), 0.0f));  // the maximum of NaN and 0 is 0
}

// Bits 0, 2, 4, 6 of x packed into bits 0..3 (Morton decode of one coordinate).
__device__ __forceinline__ int morton_even(int x) {
  x &= 0x55;
  x = (x | (x >> 1)) & 0x33;
  x = (x | (x >> 2)) & 0x0f;
  return x;
}

// Inclusive prefix of `v` over the block's threads in thread order (a block of NWARPS warps);
// `total` = block sum.
template <int NWARPS = kWarps>
__device__ __forceinline__ uint32_t block_inclusive_sum(uint32_t v, int* warp_tot, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = (int)incl;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < NWARPS; ++w) {
    const uint32_t t = (uint32_t)warp_tot[w];
    before += (w < warp) ? t : 0u;
    all += t;
  }
  __syncthreads();
  *total = all;
  return before + incl;
}

// One level of the transform over LL values held in Morton order by the lanes of a warp:
// the 2x2 block of LL grid positions (2i..2i+1, 2j..2j+1) is held by lanes
// base, base + s, base + 2s, base + 3s (a = (2i,2j), b = (2i,2j+1), c = (2i+1,2j),
// d = (2i+1,2j+1)).  The leader lane (base) keeps LL; the three details go to `upper` at
// (i, j+h), (i+h, j), (i+h, j+h) of the G x G upper block, h = the new LL side.
__device__ __forceinline__ void shuffle_level(float ll[3], int lane, int s, int m, int h, bool live,
                                              float* upper, int G) {
  float v[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    v[0][c] = __shfl_down_sync(0xffffffffu, ll[c], s);
    v[1][c] = __shfl_down_sync(0xffffffffu, ll[c], 2 * s);
    v[2][c] = __shfl_down_sync(0xffffffffu, ll[c], 3 * s);
  }
  if (live && (lane & (4 * s - 1)) == 0) {
    const int j = morton_even(m), i = morton_even(m >> 1);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float a, hl, lh, hh;
      haar4(ll[c], v[0][c], v[1][c], v[2][c], a, hl, lh, hh);
      ll[c] = a;
      upper[(i * G + j + h) * 3 + c] = hl;
      upper[((i + h) * G + j) * 3 + c] = lh;
      upper[((i + h) * G + j + h) * 3 + c] = hh;
    }
  }
}

// shuffle_level with the details stored to the batched form's upper block, laid out [channel][thread]
// (thread i * G + j owns upper-block entry (i, j)).
__device__ __forceinline__ void shuffle_level_planar(float ll[3], int lane, int s, int m, int h, bool live,
                                                      float* upf, int G) {
  float v[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    v[0][c] = __shfl_down_sync(0xffffffffu, ll[c], s);
    v[1][c] = __shfl_down_sync(0xffffffffu, ll[c], 2 * s);
    v[2][c] = __shfl_down_sync(0xffffffffu, ll[c], 3 * s);
  }
  if (live && (lane & (4 * s - 1)) == 0) {
    const int j = morton_even(m), i = morton_even(m >> 1);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float a, hl, lh, hh;
      haar4(ll[c], v[0][c], v[1][c], v[2][c], a, hl, lh, hh);
      ll[c] = a;
      upf[c * 256 + i * G + j + h] = hl;
      upf[c * 256 + (i + h) * G + j] = lh;
      upf[c * 256 + (i + h) * G + j + h] = hh;
    }
  }
}

// Geometry of one face's transform: thread t < T owns the B x B texel block at Morton(t).
template <int S>
struct FaceGeom {
  static constexpr int B = S < 4 ? S : 4;   // texel block per thread: B x B
  static constexpr int G = S / B;           // thread blocks per face side; the upper block is G x G
  static constexpr int T = G * G;           // threads holding coefficients
  static constexpr int SS = S * S;
  static constexpr int NR = B == 4 ? 15 : (B == 2 ? 3 : 0);  // coefficients held in registers
  static constexpr int NK = NR + 1;                         // plus one entry of the upper block
  static constexpr int FPI = T >= kThreads ? 1 : (kThreads / T < 6 ? kThreads / T : 6);  // faces a block holds at once
};

// Index within the face of thread tid's coefficient u (u == NR: its upper-block entry).
template <int S>
__device__ __forceinline__ int flat_in_face(int tid, int u) {
  using F = FaceGeom<S>;
  if (u == F::NR) return (tid / F::G) * S + (tid % F::G);
  int i = 0, j = 0, h = 1;
  if constexpr (F::B == 4) {
    const int bj = morton_even(tid), bi = morton_even(tid >> 1);
    const int q = u / 3;
    i = q < 4 ? 2 * bi + (q >> 1) : bi;
    j = q < 4 ? 2 * bj + (q & 1) : bj;
    h = q < 4 ? S / 2 : S / 4;
  }
  const int band = u % 3;
  return band == 0 ? i * S + j + h : (band == 1 ? (i + h) * S + j : (i + h) * S + j + h);
}

// Channel c of coefficient u < NR of thread tid's texel block, recomputed from the face at `src`
// with the same FP32 operations, in the same order, as the transform below: a level-1 detail from
// its 2x2 quad, a level-2 detail from the four quads' LL values.  The batched kernel keeps no copy
// of these coefficients; it recomputes the K winners' instead.
template <int S>
__device__ __forceinline__ float block_coef(const float* src, int tid, int u, int c) {
  using F = FaceGeom<S>;
  const int bj = morton_even(tid), bi = morton_even(tid >> 1);
  const float* blk = src + ((size_t)(F::B * bi) * S + F::B * bj) * 3 + c;
  const int q = u / 3, band = u % 3;
  auto quad = [&](int qi, int qj, float& a, float& hl, float& lh, float& hh) {
    const float* p0 = blk + ((size_t)(2 * qi) * S + 2 * qj) * 3;
    haar4(ld_stream(p0), ld_stream(p0 + 3), ld_stream(p0 + S * 3), ld_stream(p0 + S * 3 + 3), a, hl, lh, hh);
  };
  float a, hl, lh, hh;
  if (q < 4) {
    quad(q >> 1, q & 1, a, hl, lh, hh);
  } else {
    float l1[4], x, y, z;
#pragma unroll
    for (int k = 0; k < 4; ++k) quad(k >> 1, k & 1, l1[k], x, y, z);
    haar4(l1[0], l1[1], l1[2], l1[3], a, hl, lh, hh);
  }
  return band == 0 ? hl : (band == 1 ? lh : hh);
}

// The first part of the transform below: block_load loads
// thread t's B x B texel block (t < T), block_levels runs levels 1-2 on it in registers (co:
// its NR detail coefficients, ll: the block's LL value), with the same operations in the same
// order as haar_face_in_registers.
template <int S>
__device__ __forceinline__ void block_load(const float* src, int tid,
                                           float (&px)[FaceGeom<S>::B][FaceGeom<S>::B][3]) {
  using F = FaceGeom<S>;
  constexpr int B = F::B;
  if (tid >= F::T) return;
  const int bj = morton_even(tid), bi = morton_even(tid >> 1);
  const float* blk = src + ((size_t)(B * bi) * S + B * bj) * 3;
  if constexpr (B == 4) {
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float4* row = reinterpret_cast<const float4*>(blk + (size_t)r * S * 3);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const float4 v = ld_stream(row + q);
          const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) px[r][(4 * q + k) / 3][(4 * q + k) % 3] = e[k];
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 12; ++q) px[r][q / 3][q % 3] = ld_stream(blk + (size_t)r * S * 3 + q);
    }
  } else {
#pragma unroll
    for (int r = 0; r < B; ++r)
#pragma unroll
      for (int q = 0; q < 3 * B; ++q) px[r][q / 3][q % 3] = ld_stream(blk + (size_t)r * S * 3 + q);
  }
}

template <int S>
__device__ __forceinline__ void block_levels(const float (&px)[FaceGeom<S>::B][FaceGeom<S>::B][3], int tid,
                                             float (&co)[FaceGeom<S>::NR > 0 ? FaceGeom<S>::NR : 1][3],
                                             float (&ll)[3]) {
  using F = FaceGeom<S>;
  constexpr int B = F::B, NR = F::NR;
#pragma unroll
  for (int u = 0; u < (NR > 0 ? NR : 1); ++u) co[u][0] = co[u][1] = co[u][2] = 0.f;
  ll[0] = ll[1] = ll[2] = 0.f;
  if (tid >= F::T) return;
  if constexpr (B == 4) {
    float l1[2][2][3];
#pragma unroll
    for (int qi = 0; qi < 2; ++qi)
#pragma unroll
      for (int qj = 0; qj < 2; ++qj)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float a, hl, lh, hh;
          haar4(px[2 * qi][2 * qj][c], px[2 * qi][2 * qj + 1][c], px[2 * qi + 1][2 * qj][c],
                px[2 * qi + 1][2 * qj + 1][c], a, hl, lh, hh);
          l1[qi][qj][c] = a;
          const int u = (qi * 2 + qj) * 3;
          co[u][c] = hl;
          co[u + 1][c] = lh;
          co[u + 2][c] = hh;
        }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float a, hl, lh, hh;
      haar4(l1[0][0][c], l1[0][1][c], l1[1][0][c], l1[1][1][c], a, hl, lh, hh);
      ll[c] = a;
      co[12][c] = hl;
      co[13][c] = lh;
      co[14][c] = hh;
    }
  } else if constexpr (B == 2) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float a, hl, lh, hh;
      haar4(px[0][0][c], px[0][1][c], px[1][0][c], px[1][1][c], a, hl, lh, hh);
      ll[c] = a;
      co[0][c] = hl;
      co[1][c] = lh;
      co[2][c] = hh;
    }
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) ll[c] = px[0][0][c];
  }
}

// The full Haar transform of one face [S][S][3] at `src` by the block's kThreads threads:
// levels 1-2 on each thread's B x B block in registers (co: its NR detail coefficients),
// the next levels by warp shuffles, the last ones in warp 0.  The G x G upper block of the
// result (levels >= 3 and the DC term) lands in `upper` [G*G][3]; `llg` is [16][3] staging.
// Ends with a block barrier, after which `upper` is complete.
template <int S>
__device__ __forceinline__ void haar_face_in_registers(const float* src, int tid,
                                                       float (&co)[FaceGeom<S>::NR > 0 ? FaceGeom<S>::NR : 1][3],
                                                       float* upper, float* llg) {
  using F = FaceGeom<S>;
  constexpr int G = F::G;
  const int lane = tid & 31, warp = tid >> 5;
  const bool owner = tid < F::T;
  float ll[3];
  {
    float px[F::B][F::B][3];
    block_load<S>(src, tid, px);
    block_levels<S>(px, tid, co, ll);
  }
  // ---- the remaining levels over the G x G LL grid, held in Morton order by threads 0..T-1
  {
    int n = G, s = 1;  // LL grid side; lane stride between the values of one 2x2 block
#pragma unroll
    for (int lev = 0; lev < 2; ++lev)
      if (n >= 2) {
        shuffle_level(ll, lane, s, tid / (4 * s), n / 2, owner, upper, G);
        n /= 2;
        s *= 4;
      }
    if (n >= 2) {
      // at most 4 x 4 values left: leaders hand them to warp 0
      if (owner && (tid & (s - 1)) == 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) llg[(tid / s) * 3 + c] = ll[c];
      __syncthreads();
      if (warp == 0) {
        const bool live = lane < n * n;
#pragma unroll
        for (int c = 0; c < 3; ++c) ll[c] = live ? llg[lane * 3 + c] : 0.f;
        int s2 = 1;
#pragma unroll
        for (int lev = 0; lev < 2; ++lev)
          if (n >= 2) {
            shuffle_level(ll, lane, s2, lane / (4 * s2), n / 2, live, upper, G);
            n /= 2;
            s2 *= 4;
          }
        if (lane == 0)
#pragma unroll
          for (int c = 0; c < 3; ++c) upper[c] = ll[c];
      }
    } else if (tid == 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) upper[c] = ll[c];
    }
  }
  __syncthreads();
}

template <int S>
// Two CTAs per SM at most: the bound leaves the transform its registers (three per SM spilled).
__global__ void __cluster_dims__(6, 1, 1) __launch_bounds__(kThreads, 2)
    haar_topk_kernel(const float* faces, int K, int32_t* idx_out,
                     float* st_out) {
  using F = FaceGeom<S>;
  constexpr int T = F::T, SS = F::SS, NR = F::NR;
  constexpr int NW = (SS + 31) / 32;
  static_assert(T <= kThreads, "one 4x4 block per thread");

  extern __shared__ __align__(16) char smem_raw[];
  HaarSmem sm;
  smem_layout(S, K, smem_raw, &sm);
  cg::cluster_group cluster = cg::this_cluster();
  cluster.barrier_arrive();  // waited for before the first store to another CTA, which must have started
  const int face = (int)cluster.block_rank();
  const int env = blockIdx.x / 6;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool owner = tid < T;

  if (face == 0 && tid == 0) sm.scal[kScCounter] = 0;  // winner slots (read after 5 cluster barriers)
  for (int w = tid; w < NW; w += kThreads) sm.bits[w] = 0u;
  sm.hist[tid] = 0u;                     // kThreads == 256 bins
  if (tid == 0) sm.scal[kScListed] = -1;  // stays when the window holds fewer than K keys
  // (barriers in the transform order these)
  let_next_start();
  stream_wait(faces, idx_out, st_out);
  const float* src = faces + ((size_t)env * 6 + face) * (size_t)SS * 3;

  // ---- the transform: levels 1-2 in registers, the rest by shuffles and warp 0
  float co[NR > 0 ? NR : 1][3];  // detail coefficients held in registers (RGB)
  haar_face_in_registers<S>(src, tid, co, sm.upper, sm.llg);
  // ---- this thread's 16 coefficients: NR in registers, one of the upper block
  constexpr int NK = F::NK;
  auto flat_of = [&](int u) -> int { return flat_in_face<S>(tid, u); };
  uint32_t key[NK];
#pragma unroll
  for (int u = 0; u < NR; ++u) key[u] = wavelet_key_bits(co[u][0], co[u][1], co[u][2]);
  float ur = 0.f, ug = 0.f, ub = 0.f;
  if (owner) {
    ur = sm.upper[tid * 3];
    ug = sm.upper[tid * 3 + 1];
    ub = sm.upper[tid * 3 + 2];
  }
  key[NR] = wavelet_key_bits(ur, ug, ub);

  // ---- the map's largest key: every warp's to all six CTAs
  {
    uint32_t m = 0;
    if (owner)
#pragma unroll
      for (int u = 0; u < NK; ++u) m = max(m, key[u]);
    m = __reduce_max_sync(0xffffffffu, m);
    cluster.barrier_wait();
    if (lane < 6) cluster.map_shared_rank(sm.kmax, lane)[face * kWarps + warp] = m;
  }
  cluster.sync();
  uint32_t kmax = sm.kmax[lane];
  if (lane < 6 * kWarps - 32) kmax = max(kmax, sm.kmax[32 + lane]);
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  // ---- the bin of the K-th largest key in a window of 16 binades below it, at 1/16 binade (bits
  // 30..19 of the keys).  Every CTA sums the six faces' counts through distributed shared memory
  // (6 KB; it moves ~6 B per cycle: a 2,048-bin histogram of all exponents, which needs no
  // maximum, cost 8.5k cycles here), thread t the bin 255 - t.  The low half of a count is the
  // map's, the high half that of the faces before this one (24,576 keys at most: no carry).
  const int e_lo = (int)(kmax >> 23) - 15;
  auto in_window = [&](uint32_t k) { return (int)(k >> 23) >= e_lo; };
  auto bin_of = [&](uint32_t k) { return (((int)(k >> 23) - e_lo) << 4) | (int)((k >> 19) & 15u); };
  if (owner)
#pragma unroll
    for (int u = 0; u < NK; ++u)
      if (in_window(key[u])) atomicAdd(&sm.hist[bin_of(key[u])], 1u);
  cluster.sync();
  {
    const int bin = 255 - tid;
    uint32_t v[6], c = 0, all;
#pragma unroll
    for (int g = 0; g < 6; ++g) v[g] = cluster.map_shared_rank(sm.hist, g)[bin];
#pragma unroll
    for (int g = 0; g < 6; ++g) c += v[g] * (g < face ? 0x10001u : 1u);
    const uint32_t incl = block_inclusive_sum(c & 0xFFFFu, sm.warp_tot, &all), start = incl - (c & 0xFFFFu);
    sm.seg[bin] = start | (c << 16);
    sm.cur[bin] = start + (c >> 16);
    if (incl >= (uint32_t)K && start < (uint32_t)K) {
      sm.scal[kScPrefix] = (int)((uint32_t)(((e_lo + (bin >> 4)) << 4) | (bin & 15)) << 19);
      sm.scal[kScListed] = (int)incl;
    }
  }
  __syncthreads();
  const uint32_t lo_key = (uint32_t)sm.scal[kScPrefix];
  const int n_list = sm.scal[kScListed];
  if (n_list >= 0 && n_list <= list_cap(K)) {  // the same in all six CTAs
    // ---- the keys of that bin and above are listed in every CTA, bin by bin from the top (within
    // a bin by face), and each CTA ranks its own face's among their bin's; the first K are written
    if (owner)
#pragma unroll
      for (int u = 0; u < NK; ++u)
        if (key[u] >= lo_key) {
          const int32_t gflat = face * SS + flat_of(u);
          // composite key: larger key first, then smaller index first
          const uint64_t ck = ((uint64_t)key[u] << 32) | (uint64_t)(0xFFFFFFFFu - (uint32_t)gflat);
          const uint32_t slot = atomicAdd(&sm.cur[bin_of(key[u])], 1u);
#pragma unroll
          for (int g = 0; g < 6; ++g) cluster.map_shared_rank(sm.gkey, g)[slot] = ck;
          if (u < NR) sm.gval[slot] = Winner{co[u < NR ? u : 0][0], co[u < NR ? u : 0][1], co[u < NR ? u : 0][2], gflat};
          else sm.gval[slot] = Winner{ur, ug, ub, gflat};
        }
    cluster.sync();  // after it no CTA touches another's memory
    for (int e = tid; e < n_list; e += kThreads) {
      const uint64_t me = sm.gkey[e];
      const int32_t gflat = (int32_t)(0xFFFFFFFFu - (uint32_t)me);
      if (gflat / SS != face) continue;
      const uint32_t sg = sm.seg[bin_of((uint32_t)(me >> 32))];
      int rank = (int)(sg & 0xFFFFu);
      const uint64_t* o = sm.gkey + rank;
      const int n = (int)(sg >> 16);
#pragma unroll 4
      for (int i = 0; i < n; ++i) rank += o[i] > me;
      if (rank < K) {
        const Winner wv = sm.gval[e];
        const size_t out = (size_t)env * K + rank;
        idx_out[out] = wv.idx;
        st_out[out * 3 + 0] = wv.r;
        st_out[out * 3 + 1] = wv.g;
        st_out[out * 3 + 2] = wv.b;
      }
    }
    return;
  }
  cluster.sync();  // every CTA has read the histograms, whose memory the general form takes

  // ---- too many keys in that bin (ties, all zeros) or too few in the window: 4-pass radix select of the K-th largest key
  uint32_t prefix = 0, mask = 0;
  int remaining = K;
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    uint32_t* h = sm.hist + (pass & 1) * 256;
    // buffer (pass & 1) was last read remotely in pass - 2, before the previous cluster barrier
    h[tid] = 0u;
    __syncthreads();
    if (owner)
#pragma unroll
      for (int u = 0; u < NK; ++u)
        if ((key[u] & mask) == prefix) atomicAdd(&h[(key[u] >> shift) & 255u], 1u);
    cluster.sync();
    const int digit = 255 - tid;  // thread order = digits from the top
    uint32_t v[6], tot = 0;
#pragma unroll
    for (int g = 0; g < 6; ++g) v[g] = cluster.map_shared_rank(h, g)[digit];
#pragma unroll
    for (int g = 0; g < 6; ++g) tot += v[g];
    uint32_t all;
    const uint32_t incl = block_inclusive_sum(tot, sm.warp_tot, &all);
    if (incl >= (uint32_t)remaining && incl - tot < (uint32_t)remaining) {
      sm.scal[kScPrefix] = (int)(prefix | ((uint32_t)digit << shift));
      sm.scal[kScMask] = (int)(mask | (255u << shift));
      sm.scal[kScRemaining] = remaining - (int)(incl - tot);
      if (pass == 3)
#pragma unroll
        for (int g = 0; g < 6; ++g) sm.scal[kScEq + g] = (int)v[g];
    }
    __syncthreads();
    prefix = (uint32_t)sm.scal[kScPrefix];
    mask = (uint32_t)sm.scal[kScMask];
    remaining = sm.scal[kScRemaining];
  }
  // ---- ties at the threshold, taken in flat-index order (faces in order)
  const uint32_t thr = prefix;
  int eq_before = 0;
  for (int g = 0; g < face; ++g) eq_before += sm.scal[kScEq + g];
  if (owner)
#pragma unroll
    for (int u = 0; u < NK; ++u)
      if (key[u] == thr) {
        const int f = flat_of(u);
        atomicOr(&sm.bits[f >> 5], 1u << (f & 31));
      }
  __syncthreads();
  {
    uint32_t all;
    const uint32_t c = tid < NW ? (uint32_t)__popc(sm.bits[tid]) : 0u;
    const uint32_t incl = block_inclusive_sum(c, sm.warp_tot, &all);
    if (tid < NW) sm.wpre[tid] = incl - c;
  }
  __syncthreads();
  // ---- winners: slots from CTA 0's counter (one atomic per warp), stored in every CTA
  uint32_t selmask = 0;
  int n_sel = 0;
  if (owner)
#pragma unroll
    for (int u = 0; u < NK; ++u) {
      bool sel = key[u] > thr;
      if (key[u] == thr) {
        const int f = flat_of(u), w = f >> 5;
        const int rank = eq_before + (int)sm.wpre[w] + __popc(sm.bits[w] & ((1u << (f & 31)) - 1u));
        sel = rank < remaining;
      }
      if (sel) {
        selmask |= 1u << u;
        ++n_sel;
      }
    }
  int incl_w = n_sel;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl_w, o);
    if (lane >= o) incl_w += t;
  }
  int base = 0;
  if (lane == 31 && incl_w > 0) base = atomicAdd(cluster.map_shared_rank(&sm.scal[kScCounter], 0), incl_w);
  base = __shfl_sync(0xffffffffu, base, 31);
  int slot = base + incl_w - n_sel;
  if (selmask) {
#pragma unroll
    for (int u = 0; u < NK; ++u)
      if (selmask & (1u << u)) {
        const int32_t gflat = face * SS + flat_of(u);
        // composite key: larger key first, then smaller index first
        const uint64_t ck = ((uint64_t)key[u] << 32) | (uint64_t)(0xFFFFFFFFu - (uint32_t)gflat);
        Winner wv;
        if (u < NR) {
          wv = Winner{co[u][0], co[u][1], co[u][2], gflat};
        } else {
          wv = Winner{ur, ug, ub, gflat};
        }
#pragma unroll
        for (int g = 0; g < 6; ++g) {
          cluster.map_shared_rank(sm.gkey, g)[slot] = ck;
          cluster.map_shared_rank(sm.gval, g)[slot] = wv;
        }
        ++slot;
      }
  }
  cluster.sync();
  // ---- rank the K winners: CTA f takes winners f, f + 6, ...; one warp per winner
  for (int e = face + 6 * warp; e < K; e += 6 * kWarps) {
    const uint64_t me = sm.gkey[e];
    int rank = 0;
    for (int o = lane; o < K; o += 32) rank += sm.gkey[o] > me;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (lane == 0) {
      const Winner wv = sm.gval[e];
      const size_t out = (size_t)env * K + rank;
      idx_out[out] = wv.idx;
      st_out[out * 3 + 0] = wv.r;
      st_out[out * 3 + 1] = wv.g;
      st_out[out * 3 + 2] = wv.b;
    }
  }
}

// ------------------------------------------------------------------ batched form
// One persistent CTA per map at a time (no cluster): for large batches, whole maps in flight per
// SM beat the cluster's one sixth of a map each, and no step crosses an SM.
//
// Few of a map's coefficients can be among its K largest, so their keys are not kept.  The CTA
// transforms the map in six steps of a face's size, histogramming the first step's keys by their top
// 11 bits (the exponent and 3 bits of the fraction).  The K-th largest key seen so far is a lower bound
// of the K-th largest of all: a warp lists only its keys from that one's bin up, counts what it
// lists, and looks the bound up again at the third step, before it lists much of one (brighter than
// what came before), and from step to step once the list is crowded.  A step of a 64 x 64 map is an
// eighth of a face per warp, of another face each, so that the first one sees all of them: face by
// face, maps whose faces grow brighter listed too much and were read twice (each ten times brighter
// than the one before: 173 us, now 93; twice: 132, now 99).  No single copy can fetch the next step
// ahead then, which the CTAs of an SM do without (line by line: 110.7 against 107.2 us).  Taking the faces by a sample of their detail, the largest first: 112.2 us.
// No barrier guards the look-up: counts still missing only lower the bound.  When the upper levels
// are done, one block scan over the bins gives the last winner's bin, the listed keys from it up go
// to their bin's part of a second list, and each is ranked among its own bin's keys only.  Keys
// equal to 0 are never listed: a map with fewer than K others takes the first zeros by index.
//
// Levels 1-2 are thread-local; levels 3-4 (warp shuffles) leave their details in shared memory, and
// the last levels of all six faces run after one barrier, in warps 0-5.  No other coefficient is
// stored: the K winners' are recomputed from their texel blocks (block_coef).
//
// A map that overflows the first list goes over its keys once more; one whose last winner's bin is
// crowded narrows it down, as a rule by the listed keys alone (settle_list).
//
// Small faces share the block: FPI of them are transformed at once.  Bound by L1 (69% busy) and issue
// (63%): four CTAs of 64 registers fit an SM (107 us for 1,024 maps), and what they leave of the
// SM's memory as L1 matters, since a texel row's three 16-byte loads share their sectors (lists of
// 6 K + 768 keys instead of 5 K + 512 took one step of it: 110 -> 117 us).  1,024 maps, K = 300:
// 134 us -> 104 (2,950 GB/s) with all keys kept in shared memory, three scans of them and two CTAs
// per SM before; K = 64 112 -> 84, K = 1024 234 -> 200; S = 32 101 -> 46; S = 16, K = 64 70 -> 18;
// black maps 298 -> 79; small whole numbers, K = 1024 311 -> 265 (radix select over the keys of the
// map: 980).  Slower than with all keys kept: a plane gradient, whose level-2 details alone overflow
// the list, 147 -> 168 (K = 64 102 -> 136).

constexpr int kBins = 2048;       // of keys by bits 30..20
constexpr int kCtasPerSm = 4;
// Keys in the final list up to which the last winner's bin is not narrowed down: each is ranked among its
// bin's.  1,024 maps of uniform noise, K = 300: 121 us, 129 from K + 192 keys on; K = 1024: 272, 305 from
// K + K / 2 on (with settle_list a call).
__host__ __device__ constexpr int uncrowded(int K) { return K + (K > 512 ? K / 4 : 128); }
constexpr int kFineBins = 1024;   // settle_list: ten more bits; list_cap(1) composite keys hold them

__host__ __device__ constexpr int map_coeffs(int S) { return 6 * S * S; }
// Keys that may be listed while the faces pass, and in the end.
__host__ __device__ constexpr int face_list_cap(int S, int K) {
  return 5 * K + 512 < map_coeffs(S) ? 5 * K + 512 : map_coeffs(S);
}

struct BatchSmem {
  uint32_t* hist;   // [kBins + 1] counts (from the second scan on: where the bin's next key goes); then 0
  uint32_t* lkey;   // [face_list_cap] keys listed while the faces pass
  uint16_t* lid;    // [face_list_cap] their coefficient: (face * NK + u) * kThreads + thread
  uint32_t* bits;   // [6*S*S/32] in lkey's memory, after K of its entries: indices not to fill up with
  uint32_t* wpre;   // [6*S*S/32] exclusive prefix of the zeros in bits
  uint64_t* gkey;   // [list_cap] composite keys of the final list
  uint32_t* fine;   // [kFineBins] aliases gkey: counts of settle_list
  uint16_t* gid;    // [list_cap]
  uint16_t* order;  // [K] aliases lid: the winners' coefficients by rank
  uint16_t* turn;   // [K] aliases lkey: their ranks in the order they are written
  float* up;        // [6][3][kThreads] the upper-block entries: [face][channel][thread]
  float* llg;       // [6][16][3] each face's LL values left for its last levels
  int* warp_tot;
  int* scal;
};

__host__ __device__ inline size_t batch_smem_layout(int S, int K, char* base, BatchSmem* L) {
  const int nw = (map_coeffs(S) + 31) / 32;
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o = align16(o + bytes); return at; };
  const size_t oH = take(sizeof(uint32_t) * (kBins + 4));
  const size_t list = align16(sizeof(uint32_t) * face_list_cap(S, K));
  const size_t marks = sizeof(uint32_t) * 2 * nw, both = align16(sizeof(uint32_t) * K) + align16(marks);
  const size_t oL = take(list > both ? list : both), oB = o - align16(marks);
  const size_t oI = take(sizeof(uint16_t) * face_list_cap(S, K));
  const size_t oG = take(sizeof(uint64_t) * list_cap(K));
  const size_t oD = take(sizeof(uint16_t) * list_cap(K));
  const size_t oU = take(sizeof(float) * 6 * 3 * kThreads);
  const size_t oLl = take(sizeof(float) * 3 * 16 * 6);
  const size_t oW = take(sizeof(int) * kWarps);
  const size_t oS = take(sizeof(int) * 32);
  if (L) {
    L->hist = (uint32_t*)(base + oH);
    L->up = (float*)(base + oU);
    L->order = (uint16_t*)(base + oI);
    L->turn = (uint16_t*)(base + oL);
    L->lkey = (uint32_t*)(base + oL);
    L->bits = (uint32_t*)(base + oB);
    L->wpre = (uint32_t*)(base + oB) + nw;
    L->fine = (uint32_t*)(base + oG);
    L->lid = (uint16_t*)(base + oI);
    L->gkey = (uint64_t*)(base + oG);
    L->gid = (uint16_t*)(base + oD);
    L->llg = (float*)(base + oLl);
    L->warp_tot = (int*)(base + oW);
    L->scal = (int*)(base + oS);
  }
  return o;
}

// The keys of the NR detail coefficients of texel block tid (0 for u == NR and for a thread without one)
// and its block's LL value, with the operations of block_levels, two texel rows at a time.
template <int S>
__device__ __forceinline__ void face_keys(const float* src, bool owner, int tid,
                                          uint32_t (&k)[FaceGeom<S>::NK], float (&ll)[3]) {
  using F = FaceGeom<S>;
  constexpr int B = F::B;
#pragma unroll
  for (int u = 0; u < F::NK; ++u) k[u] = 0u;
  ll[0] = ll[1] = ll[2] = 0.f;
  if (!owner) return;
  const int bj = morton_even(tid), bi = morton_even(tid >> 1);
  const float* blk = src + ((size_t)(B * bi) * S + B * bj) * 3;
  if constexpr (B == 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) ll[c] = ld_stream(blk + c);
  } else {
    float l1[B == 4 ? 4 : 1][3];
    const bool vec = B == 4 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
#pragma unroll
    for (int qi = 0; qi < B / 2; ++qi) {
      float px[2][B * 3];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float* row = blk + (size_t)(2 * qi + r) * S * 3;
        if (vec) {
#pragma unroll
          for (int q = 0; q < B * 3 / 4; ++q) {
            const float4 v = ld_stream(reinterpret_cast<const float4*>(row) + q);
            px[r][4 * q] = v.x;
            px[r][4 * q + 1] = v.y;
            px[r][4 * q + 2] = v.z;
            px[r][4 * q + 3] = v.w;
          }
        } else {
#pragma unroll
          for (int q = 0; q < B * 3; ++q) px[r][q] = ld_stream(row + q);
        }
      }
#pragma unroll
      for (int qj = 0; qj < B / 2; ++qj) {
        const int q = qi * (B / 2) + qj;
        float hl[3], lh[3], hh[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
          haar4(px[0][6 * qj + c], px[0][6 * qj + 3 + c], px[1][6 * qj + c], px[1][6 * qj + 3 + c], l1[q][c], hl[c],
                lh[c], hh[c]);
        k[3 * q] = wavelet_key_bits(hl[0], hl[1], hl[2]);
        k[3 * q + 1] = wavelet_key_bits(lh[0], lh[1], lh[2]);
        k[3 * q + 2] = wavelet_key_bits(hh[0], hh[1], hh[2]);
      }
    }
    if constexpr (B == 4) {
      float hl[3], lh[3], hh[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) haar4(l1[0][c], l1[1][c], l1[2][c], l1[3][c], ll[c], hl[c], lh[c], hh[c]);
      k[12] = wavelet_key_bits(hl[0], hl[1], hl[2]);
      k[13] = wavelet_key_bits(lh[0], lh[1], lh[2]);
      k[14] = wavelet_key_bits(hh[0], hh[1], hh[2]);
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) ll[c] = l1[0][c];
    }
  }
}

// The coefficient ((face * NK + u) * kThreads + thread) at flat index g of the map: flat_in_face
// turned around.
template <int S>
__device__ __forceinline__ int id_of_flat(int g) {
  using F = FaceGeom<S>;
  constexpr int G = F::G;
  const int f = g / F::SS, i = (g % F::SS) / S, j = g % S;
  int t, u;
  if (i < G && j < G) {
    t = i * G + j;
    u = F::NR;
  } else {
    const bool second = F::B == 4 && i < S / 2 && j < S / 2;  // level 2, else level 1
    const int h = second ? S / 4 : S / 2;
    const int band = i < h ? 0 : (j < h ? 1 : 2), ii = i < h ? i : i - h, jj = j < h ? j : j - h;
    const int bi = F::B == 4 && !second ? ii / 2 : ii, bj = F::B == 4 && !second ? jj / 2 : jj;
    const int q = F::B == 4 ? (second ? 4 : (ii & 1) * 2 + (jj & 1)) : 0;
    t = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) t |= ((bj >> b & 1) << (2 * b)) | ((bi >> b & 1) << (2 * b + 1));
    u = 3 * q + band;
  }
  return (f * F::NK + u) * kThreads + t;
}

// Lower edge of the bin that holds the K-th largest key counted so far (0: fewer than K), by one
// warp: 64 bins a lane from the top, then the crossing lane's bins two a lane.
__device__ __forceinline__ uint32_t kth_bin_edge(const uint32_t* hist, int K, int lane) {
  const uint32_t h = smem_u32(hist + kBins - 64 * (lane + 1));
  uint32_t sum = 0;
#pragma unroll 4
  for (int i = 0; i < 16; ++i) {
    uint4 v;  // lanes on different banks
    asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(h + ((i + lane) & 15) * 16)
                 : "memory");
    sum += v.x + v.y + v.z + v.w;
  }
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const uint32_t hit = __ballot_sync(0xffffffffu, incl >= (uint32_t)K);
  if (!hit) return 0u;
  const int l = __ffs(hit) - 1;
  const uint32_t before = __shfl_sync(0xffffffffu, incl - sum, l);
  const int top = kBins - 64 * l - 1;
  const volatile uint32_t* hv = hist;
  const uint32_t a = hv[top - 2 * lane], b = hv[top - 2 * lane - 1];
  uint32_t in2 = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, in2, o);
    if (lane >= o) in2 += t;
  }
  const uint32_t hit2 = __ballot_sync(0xffffffffu, before + in2 >= (uint32_t)K);
  if (!hit2) return (uint32_t)(top - 63) << 20;  // counts only grow: the bin is one of these 64
  const int l2 = __ffs(hit2) - 1;
  const bool in_b = __shfl_sync(0xffffffffu, before + in2 - b < (uint32_t)K, l2);
  return (uint32_t)(top - 2 * l2 - (in_b ? 1 : 0)) << 20;
}

// The fine bin that holds the n-th largest key counted so far (-1: fewer than n), by one warp.
__device__ __forceinline__ int nth_fine_bin(const uint32_t* fine, int n, int lane) {
  const volatile uint32_t* h = fine;
  constexpr int PER = kFineBins / 32;
  uint32_t sum = 0;
#pragma unroll 8
  for (int i = 0; i < PER; ++i) sum += h[kFineBins - PER * (lane + 1) + ((i + lane) & (PER - 1))];  // other banks
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const uint32_t hit = __ballot_sync(0xffffffffu, incl >= (uint32_t)n);
  if (!hit) return -1;
  const int l = __ffs(hit) - 1, top = kFineBins - PER * l - 1;
  const uint32_t before = __shfl_sync(0xffffffffu, incl - sum, l);
  uint32_t in2 = h[top - lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, in2, o);
    if (lane >= o) in2 += t;
  }
  const uint32_t hit2 = __ballot_sync(0xffffffffu, before + in2 >= (uint32_t)n);
  return top - (hit2 ? __ffs(hit2) - 1 : 31);  // counts only grow: the bin is one of these 32
}

// Counts a warp's keys by bin, those of the first one's bin (often all: equal keys) with one atomic.
__device__ __forceinline__ void count_key(uint32_t* counts, bool in, uint32_t bin, int lane) {
  const uint32_t any = __ballot_sync(0xffffffffu, in);
  if (!any) return;
  const int lead = __ffs(any) - 1;
  const uint32_t first = __shfl_sync(0xffffffffu, bin, lead);
  const bool same = in && bin == first;
  const uint32_t n = (uint32_t)__popc(__ballot_sync(0xffffffffu, same));
  if (same ? lane == lead : in) atomicAdd(&counts[bin], same ? n : 1u);
}

// What a warp lists of the keys it forms (see above).
struct KeyList {
  const BatchSmem& sm;
  int K, cap, lane;
  uint32_t bound = 1u;   // keys of 0 are neither counted nor listed
  bool crowded = false;  // the list fills faster than faces alike would fill it

  __device__ __forceinline__ void raise() { bound = max(bound, kth_bin_edge(sm.hist, K, lane)); }

  // Lists the warp's keys k[0..N) from the bound up, and counts them unless they have been; id(u):
  // coefficient of this lane's k[u].
  template <int N, class ID>
  __device__ __forceinline__ void add(const uint32_t (&k)[N], int n_keys, bool counted, const ID& id) {
    uint32_t hits = 0;  // by u
    auto compare = [&] {
      hits = 0;
#pragma unroll
      for (int u = 0; u < N; ++u)
        if (u < n_keys) hits |= k[u] >= bound ? 1u << u : 0u;
      return (int)__reduce_add_sync(0xffffffffu, (uint32_t)__popc(hits));
    };
    int total = compare();
    if (!counted && total > max(32, K * 3 / 16)) {  // a brighter face: raise the bound before it is listed
#pragma unroll
      for (int u = 0; u < N; ++u)
        if (hits >> u & 1u) atomicAdd(&sm.hist[k[u] >> 20], 1u);
      __syncwarp();
      raise();
      total = compare();
      counted = true;
    }
    if (total == 0) return;
    // each lane's hits go side by side, after those of the lanes below it
    int at = __popc(hits);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= o) at += t;
    }
    int base = 0;
    if (lane == 31) base = atomicAdd(&sm.scal[kScListed], total);
    base = __shfl_sync(0xffffffffu, base, 31);
    crowded |= base > 4 * K + 384;
    at += base - __popc(hits);
    const bool count = !counted, room = base + total <= cap;
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (hits >> u & 1u) {
        if (room || at < cap) {
          sm.lkey[at] = k[u];
          sm.lid[at] = (uint16_t)id(u);
        }
        if (count) atomicAdd(&sm.hist[k[u] >> 20], 1u);  // also past the list's end
        ++at;
      }
  }
};

// Goes over a map's keys once more.
//  kList: lists those from lo up.
//  kMark: lists those above [lo, lo + span), clears the bits of those in it and records the least and
//         the largest of them.
//  kNarrow: counts those in [lo, lo + span) by 1/1024 of it, and lists all from the running bound up
//           that these counts give for the n-th largest of the interval.
// Keys of 0 never take part.
enum MapPass { kList, kMark, kNarrow };
template <int S, MapPass PASS>
__device__ __forceinline__ void go_over_map(const float* map, int K, uint32_t lo, int span_bits, int n) {
  using F = FaceGeom<S>;
  extern __shared__ __align__(16) char smem_raw[];
  BatchSmem sm;
  batch_smem_layout(S, K, smem_raw, &sm);
  static_assert(kFineBins / 32 == 32, "one bin a lane");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t first = max(lo, 1u), end = lo + (1u << span_bits);
  KeyList list{sm, K, face_list_cap(S, K), lane};
  list.bound = PASS == kMark ? end : first;
  const int lt = tid % F::T, fi = tid / F::T;
  uint32_t least = ~0u, most = 0u;
  __syncthreads();
  if (tid == 0) sm.scal[kScListed] = 0;
  if (PASS == kMark) {
    for (int w = tid; w < (6 * F::SS + 31) / 32; w += kThreads) sm.bits[w] = ~0u;
    if (tid == 0) sm.scal[kScLeast] = -1, sm.scal[kScMost] = 0;
  }
  if (PASS == kNarrow)
    for (int i = tid; i < kFineBins; i += kThreads) sm.fine[i] = 0u;
  __syncthreads();
#pragma unroll 1
  for (int f0 = 0; f0 < 6; f0 += F::FPI) {
    const int f = F::FPI == 1 ? (f0 + warp) % 6 : f0 + fi;  // kNarrow: the first counts see all faces
    const bool owner = fi < F::FPI && f < 6;
    uint32_t k[F::NK];
    float ll[3];
    face_keys<S>(map + (size_t)f * F::SS * 3, owner, lt, k, ll);
    const float* upf = sm.up + f * 3 * kThreads;
    if (owner) k[F::NR] = wavelet_key_bits(upf[lt], upf[kThreads + lt], upf[2 * kThreads + lt]);
    if constexpr (PASS == kNarrow) {
#pragma unroll
      for (int u = 0; u < F::NK; ++u)
        count_key(sm.fine, k[u] >= list.bound && k[u] < end, (k[u] - lo) >> (span_bits - 10), lane);
      if (f0 == 0) __syncthreads();  // without the first counts no bound
      const int b = nth_fine_bin(sm.fine, n, lane);
      if (b >= 0) list.bound = max(list.bound, lo + ((uint32_t)b << (span_bits - 10)));
    }
    list.add(k, F::NK, true, [&](int u) { return (f * F::NK + u) * kThreads + lt; });
    if constexpr (PASS == kMark) {
#pragma unroll
      for (int u = 0; u < F::NK; ++u)
        if (k[u] >= first && k[u] < end) {
          const int g = f * F::SS + flat_in_face<S>(lt, u);
          atomicAnd(&sm.bits[g >> 5], ~(1u << (g & 31)));
          least = min(least, k[u]);
          most = max(most, k[u]);
        }
    }
  }
  if constexpr (PASS == kMark) {
    least = __reduce_min_sync(0xffffffffu, least);
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) {
      atomicMin(reinterpret_cast<uint32_t*>(&sm.scal[kScLeast]), least);
      atomicMax(reinterpret_cast<uint32_t*>(&sm.scal[kScMost]), most);
    }
  }
  __syncthreads();
}

// Completes the list where the faces' pass left it incomplete or the last winner's bin crowded.
//
// A list that overflowed is made again from that bin up.  A crowded bin is narrowed down, ten bits at a time, by the listed keys or, where the list overflowed, by
// going over the map again.  This ends with the keys from a fine bin's lower edge up listed or, if a fine
// bin holds too many equal ones, with those above it listed and its own marked: they are taken in
// flat-index order.  Leaves the lower edge of the listed keys, their number and whether equal ones are
// marked in scal.  Inlined, rare as it is: around a call the kernel's 64 registers spill in every step
// (K = 64, 300 and 1024: 86.3, 106.2 and 210.5 us with a call, 83.7, 104.0 and 199.7 without).
template <int S>
__device__ __forceinline__ void settle_list(const float* map, int K) {
  extern __shared__ __align__(16) char smem_raw[];
  BatchSmem sm;
  batch_smem_layout(S, K, smem_raw, &sm);
  const int tid = threadIdx.x, lane = tid & 31, cap = face_list_cap(S, K);
  uint32_t lo = (uint32_t)sm.scal[kScPrefix];
  if (sm.scal[kScNAbove] <= uncrowded(K)) {
    go_over_map<S, kList>(map, K, lo, 0, 0);
    return;
  }
  int n_above = (int)sm.hist[lo >> 20];  // where the bin's part of the final list starts
  lo = lo >> 20 << 20;
  bool listed = sm.scal[kScListed] <= cap;  // every key from the bin up is
  for (int bits = 20; bits > 0; bits -= 10) {
    if (listed) {
      const int n_all = sm.scal[kScListed];
      __syncthreads();
      for (int i = tid; i < kFineBins; i += kThreads) sm.fine[i] = 0u;
      __syncthreads();
      for (int e0 = tid - lane; e0 < n_all; e0 += kThreads) {
        const uint32_t k = e0 + lane < n_all ? sm.lkey[e0 + lane] : 0u;
        count_key(sm.fine, k >= max(lo, 1u) && k < lo + (1u << bits), (k - lo) >> (bits - 10), lane);
      }
      __syncthreads();
    } else {
      go_over_map<S, kNarrow>(map, K, lo, bits, K - n_above);
      listed = sm.scal[kScListed] <= cap;
    }
    const int b0 = kFineBins - 4 - 4 * tid;
    const uint4 v = *reinterpret_cast<const uint4*>(sm.fine + b0);
    const uint32_t c[4] = {v.x, v.y, v.z, v.w}, sum = v.x + v.y + v.z + v.w;
    uint32_t all;
    uint32_t run = (uint32_t)n_above + block_inclusive_sum(sum, sm.warp_tot, &all) - sum;
#pragma unroll
    for (int i = 3; i >= 0; --i) {
      if (run < (uint32_t)K && run + c[i] >= (uint32_t)K) {
        sm.scal[kScPrefix] = b0 + i;
        sm.scal[kScNAbove] = (int)run;
        sm.scal[kScRemaining] = (int)c[i];
      }
      run += c[i];
    }
    __syncthreads();
    lo += (uint32_t)sm.scal[kScPrefix] << (bits - 10);
    n_above = sm.scal[kScNAbove];
    const int n = sm.scal[kScRemaining];
    __syncthreads();
    const bool fits = n_above + n <= list_cap(K);
    if (n_above + n <= uncrowded(K) || (bits == 10 && fits)) {
      if (!listed) go_over_map<S, kList>(map, K, lo, 0, 0);
      if (tid == 0) sm.scal[kScPrefix] = (int)max(lo, 1u), sm.scal[kScNAbove] = n_above + n;
      break;
    }
    if (bits == 20 && (listed || fits)) continue;
    go_over_map<S, kMark>(map, K, lo, bits - 10, 0);
    if (bits == 10 || sm.scal[kScLeast] == sm.scal[kScMost]) {
      if (tid == 0)
        sm.scal[kScPrefix] = (int)(lo + (1u << (bits - 10))), sm.scal[kScNAbove] = n_above, sm.scal[kScTied] = 1;
      break;
    }
    listed = false;  // the list holds those above only
  }
  __syncthreads();
}

template <int S>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    haar_topk_batch_kernel(const float* faces, int n_env, int K, int32_t* idx_out,
                           float* st_out) {
  using F = FaceGeom<S>;
  constexpr int T = F::T, SS = F::SS, NR = F::NR, NK = F::NK, G = F::G;
  constexpr int NL = G >= 8 ? G / 4 : 1;  // side of the LL grid left after levels 3-4
  static_assert(T <= kThreads, "one 4x4 block per thread");
  static_assert(6 * NK * kThreads <= 65536, "coefficient ids are 16-bit");
  extern __shared__ __align__(16) char smem_raw[];
  BatchSmem sm;
  batch_smem_layout(S, K, smem_raw, &sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lt = tid % T, fi = tid / T;  // texel block, and which of the FPI faces at a time
  const int cap = face_list_cap(S, K);
  float* up = sm.up;
  int* n_listed = &sm.scal[kScListed];
  stream_wait(faces, idx_out, st_out);

  for (int env = blockIdx.x; env < n_env; env += gridDim.x) {
    const float* map = faces + (size_t)env * 6 * SS * 3;
    for (int i = tid; i < kBins / 4; i += kThreads) reinterpret_cast<uint4*>(sm.hist)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) *n_listed = 0;
    __syncthreads();
    KeyList list{sm, K, cap, lane};
    for (int f0 = 0; f0 < 6; f0 += F::FPI) {
      // one face at a time: each warp its part of another one (see above)
      const int f = F::FPI == 1 ? (f0 + warp) % 6 : f0 + fi;
      const bool owner = fi < F::FPI && f < 6;
      // the next faces (after the last: this CTA's next map's first) into L2 meanwhile
      if (F::FPI > 1 && tid == 0 && (SS * 12) % 16 == 0) {
        const int n_pf = f0 + F::FPI >= 6 ? F::FPI : min(F::FPI, 6 - f0 - F::FPI);
        const long long nxt = f0 + F::FPI >= 6 ? (long long)(env + gridDim.x) * 6 : (long long)env * 6 + f0 + F::FPI;
        const float* pf = faces + (size_t)nxt * SS * 3;
        if (nxt < (long long)n_env * 6 && (reinterpret_cast<uintptr_t>(pf) & 15) == 0)
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(pf), "r"((uint32_t)(n_pf * SS * 12)) : "memory");
      }
      float* upf = up + f * 3 * kThreads;
      uint32_t k[NK];
      float ll[3];
      face_keys<S>(map + (size_t)f * SS * 3, owner, lt, k, ll);
      if (f0 == 0) {
#pragma unroll
        for (int u = 0; u < NR; ++u)
          if (k[u]) atomicAdd(&sm.hist[k[u] >> 20], 1u);
      }
      {
        int n = G, st = 1;
#pragma unroll
        for (int lev = 0; lev < 2; ++lev)
          if (n >= 2) {
            shuffle_level_planar(ll, lane, st, lt / (4 * st), n / 2, owner, upf, G);
            n /= 2;
            st *= 4;
          }
        if (n >= 2) {
          if (owner && (lt & (st - 1)) == 0)
#pragma unroll
            for (int c = 0; c < 3; ++c) sm.llg[(f * 16 + lt / st) * 3 + c] = ll[c];
        } else if (owner && lt == 0) {
#pragma unroll
          for (int c = 0; c < 3; ++c) upf[c * kThreads] = ll[c];  // the DC term
        }
        if (f0 == 0) __syncthreads();  // the first faces' counts: without them no bound
        if (NR > 0 && (f0 == 0 || f0 == 2 || list.crowded)) list.raise();
      }
      if constexpr (NR > 0) {
        list.add(k, NR, f0 == 0, [&](int u) { return (f * NK + u) * kThreads + lt; });
      }
    }
    {
      __syncthreads();  // every face's level-3/4 details and LL staging are written
      if constexpr (NL >= 2) {
        if (warp < 6) {
          const int f = warp;
          float* upf = up + f * 3 * kThreads;
          const bool live = lane < NL * NL;
          float ll[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) ll[c] = live ? sm.llg[(f * 16 + lane) * 3 + c] : 0.f;
          int n = NL, s2 = 1;
#pragma unroll
          for (int lev = 0; lev < 2; ++lev)
            if (n >= 2) {
              shuffle_level_planar(ll, lane, s2, lane / (4 * s2), n / 2, live, upf, G);
              n /= 2;
              s2 *= 4;
            }
          if (lane == 0)
#pragma unroll
            for (int c = 0; c < 3; ++c) upf[c * kThreads] = ll[c];  // the DC term
        }
        __syncthreads();  // the last levels' details are written
      }
    }
    {
      constexpr int NF = (6 + F::FPI - 1) / F::FPI;
      uint32_t k[NF];
#pragma unroll
      for (int i = 0; i < NF; ++i) {
        const int f = i * F::FPI + fi;
        const float* upf = up + f * 3 * kThreads;
        const bool owner = fi < F::FPI && f < 6;
        k[i] = owner ? wavelet_key_bits(upf[lt], upf[kThreads + lt], upf[2 * kThreads + lt]) : 0u;
      }
      list.add(k, NF, false, [&](int i) { return ((i * F::FPI + fi) * NK + NR) * kThreads + lt; });
    }
    if (tid == 0) {
      sm.scal[kScPrefix] = 1;  // every listed key, if they are fewer than K
      sm.scal[kScNAbove] = -1;
      sm.scal[kScLevels] = sm.scal[kScLevels + 1] = sm.scal[kScTied] = 0;
    }
    __syncthreads();
    // ---- the last winner's bin: eight bins a thread from the top.  A bin's part of the final list
    // starts after the keys of all bins above it.
    {
      const int b0 = kBins - 8 - 8 * tid;
      uint4* h4 = reinterpret_cast<uint4*>(sm.hist + b0);
      const uint4 lo4 = h4[0], hi4 = h4[1];
      const uint32_t c[8] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w};
      uint32_t sum = 0, all, start[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) sum += c[i];
      const uint32_t incl = block_inclusive_sum(sum, sm.warp_tot, &all);
      uint32_t run = incl - sum;
#pragma unroll
      for (int i = 7; i >= 0; --i) {
        start[i] = run;
        if (run < (uint32_t)K && run + c[i] >= (uint32_t)K) {
          sm.scal[kScPrefix] = max(1, (b0 + i) << 20);
          sm.scal[kScNAbove] = (int)(run + c[i]);
        }
        run += c[i];
      }
      h4[0] = make_uint4(start[0], start[1], start[2], start[3]);
      h4[1] = make_uint4(start[4], start[5], start[6], start[7]);
      if (tid == 0) sm.hist[kBins] = 0u;  // the end of the part above the topmost bin's
      if (tid == kThreads - 1 && all < (uint32_t)K) sm.scal[kScNAbove] = (int)all;
    }
    __syncthreads();
    if (__builtin_expect(sm.scal[kScNAbove] > uncrowded(K) || *n_listed > cap, 0)) settle_list<S>(map, K);
    const uint32_t lo_key = (uint32_t)sm.scal[kScPrefix];
    const int n_all = *n_listed, n_final = sm.scal[kScNAbove];
    for (int e = tid; e < n_all; e += kThreads) {
      const uint32_t k = sm.lkey[e];
      if (k < lo_key) continue;
      const int id = sm.lid[e], t = id % kThreads, fu = id / kThreads, f = fu / NK, u = fu % NK;
      const int g = f * SS + flat_in_face<S>(t, u);
      const uint32_t slot = atomicAdd(&sm.hist[k >> 20], 1u);
      sm.gkey[slot] = ((uint64_t)k << 32) | (uint64_t)(0xFFFFFFFFu - (uint32_t)g);
      sm.gid[slot] = (uint16_t)id;
    }
    __syncthreads();
    // one channel of a winner: its strength (and, with the first, its index)
    auto put = [&](int rank, int c, int id) {
      const int t = id % kThreads, fu = id / kThreads, f = fu / NK, u = fu % NK;
      const size_t out = (size_t)env * K + rank;
      float v = 0.f;
      if (u == NR) v = up[(f * 3 + c) * kThreads + t];
      else if constexpr (NR > 0) v = block_coef<S>(map + (size_t)f * SS * 3, t, u, c);
      if (c == 0) idx_out[out] = f * SS + flat_in_face<S>(t, u);
      st_out[out * 3 + c] = v;
    };
    for (int e = tid; e < n_final; e += kThreads) {
      const uint64_t me = sm.gkey[e];
      // its bin's part ends where the bin's next key would go, and starts where the bin above ends
      const uint32_t bin = (uint32_t)(me >> 52);
      int rank = (int)sm.hist[bin + 1];
      const uint64_t* o = sm.gkey + rank;
      const int n = (int)sm.hist[bin] - rank;
#pragma unroll 4
      for (int i = 0; i < n; ++i) rank += o[i] > me;
      if (rank < K) sm.order[rank] = sm.gid[e];
    }
    if (n_final < K) {
      // ---- then equal keys in flat-index order: those marked or, if fewer than K keys are above 0, the
      // coefficients not listed
      constexpr int NW = (6 * SS + 31) / 32, PER = (NW + kThreads - 1) / kThreads;
      if (!sm.scal[kScTied]) {
        for (int w = tid; w < NW; w += kThreads) sm.bits[w] = w * 32 + 32 <= 6 * SS ? 0u : ~0u << (6 * SS - w * 32);
        __syncthreads();
        for (int e = tid; e < n_final; e += kThreads) {
          const uint32_t g = 0xFFFFFFFFu - (uint32_t)sm.gkey[e];
          atomicOr(&sm.bits[g >> 5], 1u << (g & 31));
        }
        __syncthreads();
      }
      uint32_t mine = 0, all;
      for (int i = 0; i < PER; ++i) mine += tid * PER + i < NW ? 32u - (uint32_t)__popc(sm.bits[tid * PER + i]) : 0u;
      uint32_t run = block_inclusive_sum(mine, sm.warp_tot, &all) - mine;
      for (int i = 0; i < PER; ++i)
        if (tid * PER + i < NW) {
          sm.wpre[tid * PER + i] = run;
          run += 32u - (uint32_t)__popc(sm.bits[tid * PER + i]);
        }
      __syncthreads();
      for (int w = warp; w < NW && n_final + (int)sm.wpre[w] < K; w += kWarps) {
        const uint32_t z = ~sm.bits[w];
        const int rank = n_final + (int)sm.wpre[w] + __popc(z & ((1u << lane) - 1u));
        if ((z >> lane & 1u) && rank < K) sm.order[rank] = (uint16_t)id_of_flat<S>(w * 32 + lane);
      }
    }
    __syncthreads();
    if constexpr (F::B == 4) {
      // ---- the level-2 winners, which take four quads' texels, last: few warps then run both levels' code
      for (int i0 = warp * 32; i0 < K; i0 += kThreads) {
        const int i = i0 + lane, u = i < K ? sm.order[i] / kThreads % NK : 0;
        const bool second = u >= 12 && u < NR;
        const uint32_t in = __ballot_sync(0xffffffffu, i < K), b2 = __ballot_sync(0xffffffffu, second), b1 = in & ~b2;
        int at = 0;
        if (lane < 2) at = atomicAdd(&sm.scal[kScLevels + lane], __popc(lane ? b2 : b1));
        const int a1 = __shfl_sync(0xffffffffu, at, 0), a2 = __shfl_sync(0xffffffffu, at, 1);
        const uint32_t below = (1u << lane) - 1u;
        if (i < K) sm.turn[second ? K - 1 - a2 - __popc(b2 & below) : a1 + __popc(b1 & below)] = (uint16_t)i;
      }
      __syncthreads();
      for (int i = tid; i < 3 * K; i += kThreads) put(sm.turn[i / 3], i % 3, sm.order[sm.turn[i / 3]]);
    } else {
      for (int i = tid; i < 3 * K; i += kThreads) put(i / 3, i % 3, sm.order[i / 3]);
    }
    __syncthreads();  // the next map reuses every shared array
  }
}

// Batches of at least this many maps use the batched kernel; smaller ones the cluster form.  48
// clusters of six run at once on 148 SMs, so the cluster form's time grows every 48 maps; the
// batched kernel takes the same time for 1 to 148 maps (one per SM), which grows with K and, its
// block holding several small faces at once, falls with S.  us, cluster form and batched:
//   S = 64, K = 300    48 maps  9.0 and 24.9    96 maps 17.5 and 24.9    98 maps 23.8 and 24.9
//   S = 64, K = 1024   96 maps  26  and 41.5   128 maps 37.3 and 41.5   144 maps 47.7 and 41.8
//   S = 32, K = 300    64 maps 13.1 and 14.4    97 maps 18.6 and 14.4
//   S = 16, K = 64     32 maps  5.6 and  7.2    49 maps  9.5 and  7.2
int batch_min_maps(int S, int K) { return S <= 16 ? 49 : (K > 512 ? 129 : 97); }

template <int S>
void launch_s(const float* faces, int n_env, int K, int32_t* idx, float* strength, cudaStream_t st) {
  int dev = 0, sms = 0, max_smem = 0;
  NWPRT_CUDA(cudaGetDevice(&dev));
  NWPRT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  NWPRT_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t bsmem = batch_smem_layout(S, K, nullptr, nullptr);
  if (n_env >= batch_min_maps(S, K) && bsmem <= (size_t)max_smem) {
    NWPRT_CUDA(cudaFuncSetAttribute(haar_topk_batch_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsmem));
    int per_sm = 0;
    NWPRT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, haar_topk_batch_kernel<S>, kThreads, bsmem));
    const long long slots = (long long)sms * (per_sm > 0 ? per_sm : 1);
    const int grid = (int)(n_env < slots ? n_env : slots);
    launch_overlapped(haar_topk_batch_kernel<S>, grid, kThreads, bsmem, st, faces, n_env, K, idx, strength);
    NWPRT_CUDA(cudaGetLastError());
    return;
  }
  const size_t smem = smem_layout(S, K, nullptr, nullptr);
  NWPRT_CUDA(cudaFuncSetAttribute(haar_topk_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_overlapped(haar_topk_kernel<S>, 6LL * n_env, kThreads, smem, st, faces, K, idx, strength);
  NWPRT_CUDA(cudaGetLastError());
}

}  // namespace

size_t haar_topk_smem_bytes(int S, int K) { return smem_layout(S, K, nullptr, nullptr); }

void launch_haar_topk(const float* faces, int n_env, int S, int K, int32_t* idx, float* strength,
                      uint32_t* /*err: the kernel has no waits that could time out*/, cudaStream_t st) {
  if (n_env < 1 || n_env > (1 << 28)) fail(NWPRT_INVALID_ARG, "haar_topk: n_env out of range");
  if (S < 1 || S > kMaxS || (S & (S - 1)))
    fail(S > kMaxS ? NWPRT_UNSUPPORTED : NWPRT_INVALID_ARG,
         "haar_topk: face size must be a power of two <= 64");
  if (K < 1 || K > 6 * S * S || K > kMaxK)
    fail(NWPRT_INVALID_ARG, "haar_topk: K must be in [1, min(6*S*S, 1024)]");
  if (!faces || !idx || !strength) fail(NWPRT_INVALID_ARG, "haar_topk: null pointer");
  switch (S) {
    case 1: launch_s<1>(faces, n_env, K, idx, strength, st); break;
    case 2: launch_s<2>(faces, n_env, K, idx, strength, st); break;
    case 4: launch_s<4>(faces, n_env, K, idx, strength, st); break;
    case 8: launch_s<8>(faces, n_env, K, idx, strength, st); break;
    case 16: launch_s<16>(faces, n_env, K, idx, strength, st); break;
    case 32: launch_s<32>(faces, n_env, K, idx, strength, st); break;
    default: launch_s<64>(faces, n_env, K, idx, strength, st); break;
  }
}

}  // namespace nwprt
