// Fused plain-FP32 relight kernel: the drop-in path.
//
// A warp owns 32 (or 16) pixels for the whole pass.  Each lane encodes its pixel's position with
// the multiresolution hash grid once; then for each of the env's K wavelets the warp runs
//   cp = enc * E_k                         (ptwise_mlt, utils_kernels.h:110-127)
//   out_prd MLP -> [out_prd || aux] -> cmp_net MLP -> T_k (RGB)  (prt_network.h:73-154)
// and each lane sums += max(L_k * T_k, 0) of its pixel (computeResponse, utils_kernels.h:84-91),
// T_k staying in registers: the N x K transport matrix and the K-fold replicated input of the
// reference never exist.  Every dot product accumulates fmaf(W[j][i], x_i, .) from 0 in ascending
// i -- the order of the FP32 oracle (oracle/nwprt_oracle.c: dense_f32) -- and the K-sum is
// Kahan-compensated by default.
//
// Bound by the FP32 pipe (fma.rn.f32x2 at 2.2 issue cycles of 2.0 ideal in a register-only loop)
// and by what surrounds it.  Layout: all layer weights live in shared memory transposed to
// [in][out], the activations beside them as [row][pixel].  A layer is a small matrix product per
// warp: a thread holds 16 pixels x 4 outputs (packed pixel pairs) in registers, so a row costs it
// five 16-byte shared loads for 32 packed FMAs.  One thread per pixel, as this kernel had it,
// costs 17 loads for the same 32 (the weights are not reused): shared-memory reads bounded it.
// The warp's rows are its own, so layers need no block barrier.  The rows of a layer are unrolled
// by 32, the period of the swizzle, which leaves no address arithmetic in the loop.
// 1080p network, 611 x 407, K = 64: 28.2 -> 16.7 ms (51.3 TFLOP/s of the reference network's 53.6 kFLOP per
// evaluation, 69% of the FP32 pipe's nominal 74); 128 x 128 network, 128 x 128, K = 64: 610 -> 453 us.
#include <cmath>

#include "nwprt_internal.cuh"

namespace nwprt {
namespace {

constexpr int r4(int x) { return (x + 3) & ~3; }
constexpr int kMaxKChunk = 16;  // most wavelets whose embedding rows and strengths a block holds at a time

struct Fp32Params {
  HashLevels hl;
  const float* hash;
  const float* w;        // op_t || cn_t, transposed and padded
  int w_floats;          // multiple of 4
  const float* packed;
  const uint8_t* flag;
  const float* direct;
  const float* emb_k;
  const float* strength;
  int K;
  int k_chunk;             // blocks of 32 pixels: the wavelets held at a time (others hold kMaxKChunk)
  int64_t px_begin, n_px;  // pixel range [px_begin, n_px)
  float* indirect;
  float* with_direct;
  int clamp, kahan;
};

// Hash-grid encoding of one position (oracle/nwprt_oracle.c: orc_hash_encode_f32); feature i to put(i, v).
template <class PUT>
__device__ __forceinline__ void hash_encode(const HashLevels& hl, const float* __restrict__ table, float px, float py,
                                            float pz, const PUT& put) {
  const float p[3] = {fminf(fmaxf(px, 0.f), 1.f), fminf(fmaxf(py, 0.f), 1.f),
                      fminf(fmaxf(pz, 0.f), 1.f)};
  const int F = hl.n_features;
  for (int l = 0; l < hl.n_levels; ++l) {
    const int N = hl.res[l];
    uint32_t i0[3];
    float w[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float xl = __fmul_rn(p[d], (float)N);
      int i = (int)floorf(xl);
      if (i > N - 1) i = N - 1;
      i0[d] = (uint32_t)i;
      w[d] = __fsub_rn(xl, (float)i);
    }
    const uint32_t N1 = (uint32_t)N + 1u;
    const bool dense = (hl.dense_mask >> l) & 1u;
    const uint32_t T = hl.size[l];
    const float* lvl = table + (size_t)hl.offset[l] * F;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint32_t bx = c & 1, by = (c >> 1) & 1, bz = (c >> 2) & 1;
      const float wx = bx ? w[0] : __fsub_rn(1.f, w[0]);
      const float wy = by ? w[1] : __fsub_rn(1.f, w[1]);
      const float wz = bz ? w[2] : __fsub_rn(1.f, w[2]);
      const float wc = __fmul_rn(__fmul_rn(wx, wy), wz);
      const uint32_t x = i0[0] + bx, y = i0[1] + by, z = i0[2] + bz;
      const uint32_t e = dense ? x + y * N1 + z * N1 * N1
                               : ((x ^ (y * 2654435761u) ^ (z * 805459861u)) & (T - 1u));
      const float* th = lvl + (size_t)e * F;
      if (F == 2) {
        const float2 v = __ldg(reinterpret_cast<const float2*>(th));
        acc[0] = fmaf(wc, v.x, acc[0]);
        acc[1] = fmaf(wc, v.y, acc[1]);
      } else {
        for (int f = 0; f < F; ++f) acc[f] = fmaf(wc, __ldg(th + f), acc[f]);
      }
    }
    for (int f = 0; f < F; ++f) put(l * F + f, acc[f]);
  }
}

// Two FP32 values in one 64-bit register, and the packed FMA of sm_100 on such pairs:
// fma.rn.f32x2 rounds each lane once, exactly as fmaf does, so a pair of output neurons
// accumulated side by side keeps the oracle's bits with half the FMA instructions.
__device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void f2_fma(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// ---- the network: its layer sequence, read at run time.  Output widths up to kMaxOut.
constexpr int kMaxOut = 64;
constexpr int kMaxNetLayers = 2 * kMaxLayers;
struct NetLayer {
  int in, out, relu, mode;  // 0: the activation rows; 1: the CP product; 2: [out_prd || aux]
  int w_off;                // float offset of the [in][w_stride] block
};
struct NetSeq {
  NetLayer l[kMaxNetLayers];
  int n = 0;
  // rows of the activation array: hidden activations (and the CP product) from 0, aux values from
  // aux (a multiple of 32), hash features from enc
  int enc = 0, aux = 0, rows = 0, opo = 0, d = 0, auxw = 0;
};

// Activations of a block's NT pixels, [row][NT] in shared memory.  Within each 128-byte line of
// 32 pixels the eight 16-byte chunks are XOR-swizzled by row / 4, so that neither the tile reads
// (one row, a few pixel groups) nor the tile writes (output groups of four rows, one pixel group)
// meet a bank conflict.  px: pixel within the line.
template <int NT>
__device__ __forceinline__ int act_at(int row, int px) {
  return row * NT + ((((px >> 2) ^ (row >> 2)) & 7) << 2) + (px & 3);
}

// acc += W[:, i] x_i for rows row0 .. row0 + n of the activations, in ascending order (row0: a
// multiple of 32).  A thread holds PX pixels (from px0 of its line; pixel pairs packed) x 4
// outputs.  w: the first weight row at the thread's outputs, rows WS floats apart.
template <int PX, int WS, int NT>
__device__ __forceinline__ void mm_rows(unsigned long long (&acc)[4][PX / 2], const float* __restrict__ w,
                                        const float* act, int row0, int n, int px0) {
  constexpr int C = PX / 4;  // 16-byte chunks of a thread's pixels in a row
  auto step = [&](const float* wr, const float* xr, int swz) {
    unsigned long long xp[PX / 2];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      // (px0 / 4 + c) ^ swz, px0 / 4 being a multiple of C
      const float4 v = *reinterpret_cast<const float4*>(xr + (((px0 >> 2) ^ (swz & ~(C - 1))) << 2) +
                                                        ((c ^ (swz & (C - 1))) << 2));
      xp[2 * c] = f2_pack(v.x, v.y);
      xp[2 * c + 1] = f2_pack(v.z, v.w);
    }
    const float4 v = *reinterpret_cast<const float4*>(wr);
    const unsigned long long wd[4] = {f2_pack(v.x, v.x), f2_pack(v.y, v.y), f2_pack(v.z, v.z), f2_pack(v.w, v.w)};
#pragma unroll
    for (int o = 0; o < 4; ++o)
#pragma unroll
      for (int c = 0; c < PX / 2; ++c) f2_fma(acc[o][c], wd[o], xp[c]);
  };
  const float* x = act + row0 * NT;
#pragma unroll 1
  for (; n >= 32; n -= 32, x += 32 * NT, w += 32 * WS) {
#pragma unroll
    for (int i = 0; i < 32; ++i) step(w + i * WS, x + i * NT, i >> 2);
  }
  int i = 0;
#pragma unroll 1
  for (; i + 8 <= n; i += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) step(w + (i + u) * WS, x + (i + u) * NT, (i + u) >> 2);
  }
#pragma unroll 1
  for (; i < n; ++i) step(w + i * WS, x + i * NT, i >> 2);
}

// Width of a weight row in shared memory: what the output groups of dense_tile cover, or one
// 16-byte load of the output layer.
constexpr int w_stride(int out, bool output_layer) {
  return output_layer ? r4(out) : out <= 32 ? 32 : out <= 64 ? 64 : r4(out);
}

// One hidden layer of a warp's WP pixels, in place in the activation rows.  OG output groups of 4
// outputs (16 for layers of 33 to 64 outputs, else 8) x 32 / OG pixel groups.
template <int OG, int WP, int NT>
__device__ __forceinline__ void dense_tile(const NetLayer& L, const NetSeq& g, const float* __restrict__ W, float* act,
                                           int lane, int line_px) {
  constexpr int PX = WP * OG / 32, C = PX / 4;
  const int px0 = line_px + lane / OG * PX, og = lane & (OG - 1);
  unsigned long long acc[4][PX / 2];
#pragma unroll
  for (int o = 0; o < 4; ++o)
#pragma unroll
    for (int c = 0; c < PX / 2; ++c) acc[o][c] = 0ull;
  const float* w = W + og * 4;
  int row0 = 0, n = L.mode == 2 ? g.opo : L.in;
#pragma unroll 1  // one copy of the unrolled rows in the instruction cache
  for (int left = L.in; left > 0; n = left, row0 = g.aux) {
    mm_rows<PX, OG * 4, NT>(acc, w, act, row0, n, px0);
    w += n * (OG * 4);
    left -= n;
  }
  __syncwarp();  // every read of the rows below is done
  float* dst = act + og * 4 * NT;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int at = (((px0 >> 2) ^ (og & 7 & ~(C - 1))) << 2) + ((c ^ (og & (C - 1))) << 2);
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      float4 v;
      f2_unpack(acc[o][2 * c], v.x, v.y);
      f2_unpack(acc[o][2 * c + 1], v.z, v.w);
      if (L.relu) v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
      *reinterpret_cast<float4*>(dst + o * NT + at) = v;
    }
  }
  __syncwarp();
}

// The 3-wide output layer over rows row0 .. row0 + n (row0: a multiple of 32), one pixel per lane.
template <int NT>
__device__ __forceinline__ void out_rows(float (&T)[3], const float* __restrict__ w, const float* act, int row0, int n,
                                         int px) {
  auto step = [&](const float* wr, const float* xr, int swz) {
    const float x = xr[(((px >> 2) ^ swz) << 2) + (px & 3)];
    const float4 v = *reinterpret_cast<const float4*>(wr);
    T[0] = fmaf(v.x, x, T[0]);
    T[1] = fmaf(v.y, x, T[1]);
    T[2] = fmaf(v.z, x, T[2]);
  };
  const float* x = act + row0 * NT;
#pragma unroll 1
  for (; n >= 32; n -= 32, x += 32 * NT, w += 32 * 4) {
#pragma unroll
    for (int i = 0; i < 32; ++i) step(w + i * 4, x + i * NT, i >> 2);
  }
#pragma unroll 2
  for (int i = 0; i < n; ++i) step(w + i * 4, x + i * NT, i >> 2);
}

// NT pixels per block, WP per warp.
template <int NT, int WP>
__global__ void __launch_bounds__(NT / WP * 32, 1) relight_fp32_kernel(const __grid_constant__ Fp32Params p,
                                                                       const __grid_constant__ NetSeq g) {
  constexpr int kThreads = NT / WP * 32;
  extern __shared__ __align__(16) float sm[];
  float* sW = sm;
  float* sE = sW + p.w_floats;
  const int k_chunk = NT == 32 ? p.k_chunk : kMaxKChunk;  // a constant where it can be: 0.5% of the pass
  float* sL = sE + r4(k_chunk * g.d);
  float* sAct = sL + k_chunk * 4;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int i = tid * 4; i < p.w_floats; i += kThreads * 4)
    *reinterpret_cast<float4*>(sW + i) = __ldg(reinterpret_cast<const float4*>(p.w + i));
  // the warp's pixels: WP of a line; lanes beyond WP repeat one and store nothing
  const int warp_px = (tid >> 5) * WP, line_px = warp_px & 31, lpx = lane & (WP - 1);
  float* act = sAct + (warp_px & ~31);
  const int64_t px = p.px_begin + (int64_t)blockIdx.x * NT + warp_px + lpx;
  const bool valid = px < p.n_px;
  const bool active = valid && p.flag[px] != 0;
  const bool warp_active = __any_sync(0xffffffffu, active);
  if (lane < WP) {
    // a pixel that is not active is evaluated (with zeros) beside its warp's others, and not summed
    if (active) {
      const float4* row = reinterpret_cast<const float4*>(p.packed) + px * 4;
      const float4 r0 = row[0], r1 = row[1], r2 = row[2], r3 = row[3];
      hash_encode(p.hl, p.hash, r0.x, r0.y, r0.z,
                  [&](int i, float v) { act[act_at<NT>(g.enc + i, line_px + lpx)] = v; });
      const float aux13[13] = {r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, r2.z, r2.w, r3.x, r3.y, r3.z, r3.w};
      for (int i = 0; i < g.auxw; ++i) act[act_at<NT>(g.aux + i, line_px + lpx)] = i < 13 ? aux13[i] : 1.0f;
    } else {
      for (int i = 0; i < g.d; ++i) act[act_at<NT>(g.enc + i, line_px + lpx)] = 0.f;
      for (int i = 0; i < g.auxw; ++i) act[act_at<NT>(g.aux + i, line_px + lpx)] = 0.f;
    }
  }
  float s[3] = {0.f, 0.f, 0.f}, comp[3] = {0.f, 0.f, 0.f};
  for (int k0 = 0; k0 < p.K; k0 += k_chunk) {
    const int kc = min(k_chunk, p.K - k0);
    __syncthreads();
    for (int i = tid; i < kc * g.d; i += kThreads) sE[i] = p.emb_k[(size_t)k0 * g.d + i];
    for (int i = tid; i < kc * 3; i += kThreads) sL[(i / 3) * 4 + i % 3] = p.strength[(size_t)k0 * 3 + i];
    __syncthreads();
    if (!warp_active) continue;
    for (int kk = 0; kk < kc; ++kk) {
      // cp_i = enc_i * E_k,i (ptwise_mlt) into the first rows
      const float* e = sE + kk * g.d;
#pragma unroll 8
      for (int i = lane / WP; i < g.d; i += 32 / WP)
        act[act_at<NT>(i, line_px + lpx)] = __fmul_rn(act[act_at<NT>(g.enc + i, line_px + lpx)], e[i]);
      __syncwarp();
#pragma unroll 1
      for (int li = 0; li + 1 < g.n; ++li) {
        const NetLayer& L = g.l[li];
        if (L.out > 32) dense_tile<16, WP, NT>(L, g, sW + L.w_off, act, lane, line_px);
        else dense_tile<8, WP, NT>(L, g, sW + L.w_off, act, lane, line_px);
      }
      float T[3] = {0.f, 0.f, 0.f};
      {
        const NetLayer& L = g.l[g.n - 1];
        const float* w = sW + L.w_off;
        int row0 = 0, n = L.mode == 2 ? g.opo : L.in;
#pragma unroll 1
        for (int left = L.in; left > 0; n = left, row0 = g.aux) {
          out_rows<NT>(T, w, act, row0, n, line_px + lpx);
          w += n * 4;
          left -= n;
        }
      }
      if (active) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float term = __fmul_rn(sL[kk * 4 + c], T[c]);
          if (p.clamp) term = fmaxf(term, 0.0f);
          if (p.kahan) {
            const float y = __fsub_rn(term, comp[c]);
            const float t = __fadd_rn(s[c], y);
            comp[c] = __fsub_rn(__fsub_rn(t, s[c]), y);
            s[c] = t;
          } else {
            s[c] = __fadd_rn(s[c], term);
          }
        }
      }
      __syncwarp();  // the output layer's reads, before the next wavelet's first writes
    }
  }
  if (valid && lane < WP) {
    const float4 dl = reinterpret_cast<const float4*>(p.direct)[px];
    reinterpret_cast<float4*>(p.indirect)[px] = make_float4(s[0], s[1], s[2], 1.f);
    reinterpret_cast<float4*>(p.with_direct)[px] =
        make_float4(__fadd_rn(s[0], dl.x), __fadd_rn(s[1], dl.y), __fadd_rn(s[2], dl.z), 1.f);
  }
}

// The layer sequence of d: out_prd's layers (the first takes the CP product), then cmp_net's
// (the first takes [out_prd || aux]); the last layer writes T.
bool net_seq(const NetDims& d, int max_smem, NetSeq* g, std::string* why) {
  auto no = [&](const char* m) { if (why) *why = m; return false; };
  if (d.op_nl + d.cn_nl > kMaxNetLayers) return no("fp32 relight: too many layers");
  int off = 0, widest = d.op_out;
  for (int i = 0; i < d.op_nl; ++i) {
    if (d.op_outs[i] > kMaxOut) return no("fp32 relight: layer widths above 64 are not supported");
    g->l[g->n++] = NetLayer{d.op_in[i], d.op_outs[i], i + 1 < d.op_nl ? 1 : 0, i == 0 ? 1 : 0, off};
    off += d.op_in[i] * w_stride(d.op_outs[i], false);
    widest = d.op_outs[i] > widest ? d.op_outs[i] : widest;
  }
  for (int i = 0; i < d.cn_nl; ++i) {
    if (d.cn_outs[i] > kMaxOut) return no("fp32 relight: layer widths above 64 are not supported");
    g->l[g->n++] = NetLayer{d.cn_in[i], d.cn_outs[i], i + 1 < d.cn_nl ? 1 : 0, i == 0 ? 2 : 0, off};
    off += d.cn_in[i] * w_stride(d.cn_outs[i], i + 1 == d.cn_nl);
    if (i + 1 < d.cn_nl) widest = d.cn_outs[i] > widest ? d.cn_outs[i] : widest;
  }
  if (d.cn_outs[d.cn_nl - 1] != 3) return no("fp32 relight: cmp_net must end in 3 outputs");
  // The largest network: its weights beside the activations of 128 pixels, nothing padded.
  size_t floats = (size_t)kMaxKChunk * (d.enc_dims() + 4) + (size_t)128 * (widest + d.enc_dims() + d.aux_width);
  for (int i = 0; i < d.op_nl; ++i) floats += (size_t)d.op_in[i] * r4(d.op_outs[i]);
  for (int i = 0; i < d.cn_nl; ++i) floats += (size_t)d.cn_in[i] * r4(d.cn_outs[i]);
  if (floats * sizeof(float) > (size_t)max_smem) return no("fp32 relight: network too large for shared memory");
  g->d = d.enc_dims();
  g->opo = d.op_out;
  g->auxw = d.aux_width;
  if (g->d > widest) widest = g->d;  // the CP product takes the first rows
  g->aux = (widest + 31) & ~31;
  g->enc = g->aux + g->auxw;
  g->rows = g->enc + g->d;
  return true;
}

size_t net_smem_bytes(const NetSeq& g, int w_floats, int nt, int k_chunk) {
  return sizeof(float) * ((size_t)w_floats + r4(k_chunk * g.d) + k_chunk * 4 + (size_t)g.rows * nt);
}

template <int NT, int WP>
void launch_nt(const Fp32Params& p, const NetSeq& g, cudaStream_t st) {
  auto k = relight_fp32_kernel<NT, WP>;
  const size_t smem = net_smem_bytes(g, p.w_floats, NT, p.k_chunk);
  NWPRT_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t n = p.n_px - p.px_begin;
  k<<<(unsigned)((n + NT - 1) / NT), NT / WP * 32, smem, st>>>(p, g);
  NWPRT_CUDA(cudaGetLastError());
}

}  // namespace

// Transposes each row-major [out][in] layer to [in][w_stride] (zero padded).
void pack_fp32_weights(const NetDims& d, const float* op, const float* cn, std::vector<float>* op_t,
                       std::vector<float>* cn_t) {
  auto pack = [](int nl, const int* in, const int* out, const float* src, std::vector<float>* dst, bool ends) {
    dst->clear();
    for (int l = 0; l < nl; ++l) {
      const int o4 = w_stride(out[l], ends && l + 1 == nl);
      size_t base = dst->size();
      dst->resize(base + (size_t)in[l] * o4, 0.f);
      for (int j = 0; j < out[l]; ++j)
        for (int i = 0; i < in[l]; ++i) (*dst)[base + (size_t)i * o4 + j] = src[(size_t)j * in[l] + i];
      src += (size_t)in[l] * out[l];
    }
  };
  pack(d.op_nl, d.op_in, d.op_outs, op, op_t, false);
  pack(d.cn_nl, d.cn_in, d.cn_outs, cn, cn_t, true);
}

// Any network that net_seq accepts.
void launch_relight_fp32(const NetDims& d, const HashLevels& hl, const DeviceWeights& w,
                         const RelightJob& job, int clamp, int kahan, cudaStream_t st) {
  if (job.n_px <= job.px_begin) return;
  Fp32Params p;
  p.hl = hl;
  p.hash = w.hash;
  p.w = w.op_t;  // op_t and cn_t are stored back to back
  p.w_floats = (int)(w.op_t_floats + w.cn_t_floats);
  p.packed = job.packed;
  p.flag = job.flag;
  p.direct = job.direct;
  p.emb_k = job.emb_k;
  p.strength = job.strength;
  p.K = job.K;
  p.px_begin = job.px_begin;
  p.n_px = job.n_px;
  p.indirect = job.indirect;
  p.with_direct = job.with_direct;
  p.clamp = clamp;
  p.kahan = kahan;
  int dev = 0, max_smem = 0, sms = 0;
  NWPRT_CUDA(cudaGetDevice(&dev));
  NWPRT_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  NWPRT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  NetSeq g;
  std::string why;
  if (!net_seq(d, max_smem, &g, &why)) fail(NWPRT_UNSUPPORTED, why);
  const NetLayer& last = g.l[g.n - 1];
  if (last.w_off + last.in * w_stride(last.out, true) != p.w_floats) fail(NWPRT_INVALID_ARG, "fp32 weight layout mismatch");
  const int64_t n = p.n_px - p.px_begin;
  p.k_chunk = kMaxKChunk;
  auto fits = [&](int nt) { return net_smem_bytes(g, p.w_floats, nt, p.k_chunk) <= (size_t)max_smem; };
  // Pixels per block (mostly one block per SM at a time, as its weights and activations fill the
  // shared memory).  Blocks of 256 and more give a warp 32 pixels, smaller ones 16: half the
  // arithmetic per weight read, twice the warps.  us of one round of 148 blocks at K = 64:
  //   pixels           64    128    256    384    512
  //   128x128 network  306    457    826   1136   1498
  //   1080p network    764   1261   2460   (the last two do not fit)
  // The launch takes the size whose rounds cost least, by the first row's ratios.
  struct Form { int nt; double cost; };
  const Form forms[] = {{512, 1498}, {384, 1136}, {256, 826}, {128, 457}, {64, 306}};
  int nt = 0;
  double best = 0;
  for (const Form& f : forms) {
    if (!fits(f.nt)) continue;
    const double c = (double)(((n + f.nt - 1) / f.nt + sms - 1) / sms) * f.cost;
    if (!nt || c < best) nt = f.nt, best = c;
  }
  if (!nt) {
    // A block of 32 pixels, with as many wavelets at a time as fit.  Padded weight rows can take more
    // than the smaller block saves (two deep networks 33 to 46 wide behind some 160 hash features and
    // more), but one wavelet at a time fits every network that net_seq accepts.
    while (p.k_chunk > 1 && !fits(32)) p.k_chunk /= 2;
    if (fits(32)) nt = 32;
  }
  switch (nt) {
    case 512: launch_nt<512, 32>(p, g, st); break;
    case 384: launch_nt<384, 32>(p, g, st); break;
    case 256: launch_nt<256, 32>(p, g, st); break;
    case 128: launch_nt<128, 16>(p, g, st); break;
    case 64: launch_nt<64, 16>(p, g, st); break;
    case 32: launch_nt<32, 16>(p, g, st); break;
    default: fail(NWPRT_UNSUPPORTED, "fp32 relight: network too large for shared memory");
  }
}

}  // namespace nwprt
