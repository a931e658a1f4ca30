// RMS-norm (replaces rms_norm_kernel, include/rdna4/nn.cuh:23-63 and rms_norm_launch,
// :239-243 of the reference) and the fused pre-attention stage of a full-attention
// layer: what Graph::full_attn does in seven launches between the projections and
// the attention call (include/rdna4/graph.cuh:915-954) --
//   deinterleave [q | gate] per head, RMS-norm of every q and k head row with its weight,
//   partial RoPE of q and k, quantize-and-store of the k and v rows into the caches --
// in ONE launch, one warp per 256-wide head row (up to eight tokens: one per 32-value block of a K or V row).
//
// The sum of squares keeps the reference kernel's order (256 threads each squaring one
// element, then a shared-memory tree over strides 128 .. 1), so it is bit-identical to
// it; rsqrt is the correctly rounded 1 / sqrt (the reference's device intrinsic is
// approximate). A warp lane L holds elements L, L+32, .. L+224 of the row, which makes
// the first three tree levels and the RoPE pairs (p, p + n_rot/2 with n_rot/2 a multiple
// of 32) lane-local and gives the quantizer its native layout (lane j = element j of a
// 32-value block).
#include "rd_common.cuh"
#include "rd_internal.h"
#include "rd_quant.cuh"

namespace rd {

constexpr int kRmsThreads = 256;

__global__ void __launch_bounds__(kRmsThreads)
rms_norm_kernel(const float *__restrict__ x, const float *__restrict__ w, float *__restrict__ y,
                int64_t ncols, float eps) {
  __shared__ float partial[kRmsThreads];
  pdl_launch_dependents();
  pdl_wait();
  const float *xr = x + (int64_t)blockIdx.x * ncols;
  float *yr = y + (int64_t)blockIdx.x * ncols;
  float acc = 0.0f;
  for (int64_t i = threadIdx.x; i < ncols; i += kRmsThreads) acc = __fmaf_rn(xr[i], xr[i], acc);
  partial[threadIdx.x] = acc;
  __syncthreads();
  for (int stride = kRmsThreads / 2; stride > 0; stride >>= 1) {
    if ((int)threadIdx.x < stride)
      partial[threadIdx.x] = __fadd_rn(partial[threadIdx.x], partial[threadIdx.x + stride]);
    __syncthreads();
  }
  const float scale =
      __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(partial[0], (float)ncols), eps)));
  for (int64_t i = threadIdx.x; i < ncols; i += kRmsThreads) {
    const float v = __fmul_rn(xr[i], scale);
    yr[i] = w != nullptr ? __fmul_rn(v, w[i]) : v;
  }
}

int launch_rms_norm(const float *x, const float *w, float *y, int64_t nrows, int64_t ncols, float eps,
                    cudaStream_t st) {
  if (nrows == 0) return RD_OK;
  return launch_pdl(8, rms_norm_kernel, dim3((unsigned)nrows), dim3(kRmsThreads), 0, st, x, w, y, ncols, eps) ==
                 cudaSuccess
             ? RD_OK
             : RD_ERR_CUDA;
}

struct PreAttnArgs {
  const float *qg;      // [n_tok][n_head][2 * 256]: q then gate per head
  const float *k_src;   // [n_tok][nkv][256]
  const float *v_src;   // [n_tok][nkv][256]
  const float *q_w;     // [256] or null
  const float *k_w;     // [256] or null
  float *q_out;         // [n_tok][n_head][256]
  float *gate_out;      // [n_tok][n_head][256]
  uint8_t *k_rows;      // cache rows of the n_tok new tokens, [n_tok][nkv] rows
  uint8_t *v_rows;
  const int32_t *pos;   // [n_tok]
  int n_tok, n_head, nkv, n_rot;
  float eps, freq_base;
  RopeTable rope;
};

// Frequencies beyond the table (n_rot above 128): kept out of line, the common path stays short.
__device__ __noinline__ float rope_freq_slow(float freq_base, int p, int n_rot) {
  return (float)pow((double)freq_base, (double)(-2.0f * (float)p / (float)n_rot));
}

// Normalise (optional) and rotate the 8 values a lane holds of one head row; wv holds the
// lane's norm weights.
__device__ __forceinline__ void norm_rope_row(float (&x)[8], const float (&wv)[8], bool weighted, float eps,
                                              int n_rot, float fpos, const RopeTable &tab,
                                              float freq_base, int lane) {
  float p[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) p[k] = __fmul_rn(x[k], x[k]);
#pragma unroll
  for (int k = 0; k < 4; ++k) p[k] = __fadd_rn(p[k], p[k + 4]);   // stride 128
  p[0] = __fadd_rn(p[0], p[2]);                                   // stride 64
  p[1] = __fadd_rn(p[1], p[3]);
  float s = __fadd_rn(p[0], p[1]);                                // stride 32
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_down_sync(0xffffffffu, s, o));
  s = __shfl_sync(0xffffffffu, s, 0);
  const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(s, (float)kHeadDim), eps)));
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    x[k] = __fmul_rn(x[k], scale);
    if (weighted) x[k] = __fmul_rn(x[k], wv[k]);
  }
  const int hk = n_rot / 64;   // registers per half: pairs (k, k + hk), k < hk
#pragma unroll 1
  for (int k = 0; k < hk; ++k) {
    const int pidx = lane + 32 * k;
    const float freq = pidx < kRopeTablePairs ? tab.f[pidx] : rope_freq_slow(freq_base, pidx, n_rot);
    float c, sn;
    sincosf(fpos * freq, &sn, &c);
    // x[k] and x[k + hk] by value: the loop stays rolled (one sincosf in the code) and x in registers
    float x0 = 0.f, x1 = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      x0 = i == k ? x[i] : x0;
      x1 = i == k + hk ? x[i] : x1;
    }
    const float y0 = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, sn));
    const float y1 = __fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, c));
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = i == k ? y0 : i == k + hk ? y1 : x[i];
  }
}

// SPLIT (a decode step or a verify block): latency-bound, so a warp quantizes ONE 32-value
// block -- the eight blocks of a K row are eight warps that each load and normalise the whole
// row (its sum of squares needs it; the loads hit L1 / L2) -- and everything a row needs is
// requested before anything is used. At one token that is 88 short warps over 22 CTAs where one
// warp per row ran eight quantizations in sequence on 4 SMs, in code eight times as long
// (instruction fetch is a large part of a kernel that runs once): a 16-layer step over 137 f16
// keys 253 -> 240 us, over 4096 keys 350 -> 294 us. Without SPLIT (prompt chunks) a warp owns a whole row.
constexpr int kPreSplitTokens = 8;
template <int KT, int VT, bool SPLIT>
__global__ void __launch_bounds__(256) pre_attn_kernel(const __grid_constant__ PreAttnArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int kv_warps = SPLIT ? 8 * a.nkv : a.nkv;   // per tensor
  const int per_tok = a.n_head + 2 * kv_warps;
  pdl_launch_dependents();
  pdl_wait();
  if (row >= (int64_t)a.n_tok * per_tok) return;
  const int tok = (int)(row / per_tok);
  int r = (int)(row % per_tok);
  if (r >= a.n_head + kv_warps) {   // a V row, or one block of it
    r -= a.n_head + kv_warps;
    const int kvh = SPLIT ? r >> 3 : r;
    const float *src = a.v_src + ((size_t)tok * a.nkv + kvh) * kHeadDim;
    uint8_t *dst = a.v_rows + ((size_t)tok * a.nkv + kvh) * row_bytes(VT);
    if (SPLIT) {
      store_block<VT>(src[lane + 32 * (r & 7)], dst, r & 7, lane);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) store_block<VT>(src[lane + 32 * k], dst, k, lane);
    }
    return;
  }
  const bool is_q = r < a.n_head;
  const int kvh = SPLIT ? (r - a.n_head) >> 3 : r - a.n_head;
  const float *src = is_q ? a.qg + ((size_t)tok * a.n_head + r) * (2 * kHeadDim)
                          : a.k_src + ((size_t)tok * a.nkv + kvh) * kHeadDim;
  const float *w = is_q ? a.q_w : a.k_w;
  const float fpos = (float)a.pos[tok];
  float x[8], wv[8], gv[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    x[k] = src[lane + 32 * k];
    wv[k] = w != nullptr ? w[lane + 32 * k] : 1.f;
    gv[k] = is_q ? src[kHeadDim + lane + 32 * k] : 0.f;
  }
  norm_rope_row(x, wv, w != nullptr, a.eps, a.n_rot, fpos, a.rope, a.freq_base, lane);
  if (is_q) {
    // a query head: the gate split off, the row normalised and rotated
    float *qo = a.q_out + ((size_t)tok * a.n_head + r) * kHeadDim;
    float *go = a.gate_out + ((size_t)tok * a.n_head + r) * kHeadDim;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      qo[lane + 32 * k] = x[k];
      go[lane + 32 * k] = gv[k];
    }
  } else {
    uint8_t *dst = a.k_rows + ((size_t)tok * a.nkv + kvh) * row_bytes(KT);
    if (SPLIT) {
      const int blk = (r - a.n_head) & 7;
      float v = x[0];
#pragma unroll
      for (int k = 1; k < 8; ++k) v = k == blk ? x[k] : v;
      store_block<KT>(v, dst, blk, lane);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) store_block<KT>(x[k], dst, k, lane);
    }
  }
}

template <int KT>
static int pre_attn_v(int vt, const PreAttnArgs &a, cudaStream_t st) {
  const bool split = a.n_tok <= kPreSplitTokens;
  const int64_t warps = (int64_t)a.n_tok * (a.n_head + 2 * (split ? 8 : 1) * a.nkv);
  const int per_cta = split ? 4 : 8;
  const dim3 grid((unsigned)((warps + per_cta - 1) / per_cta)), block(32 * per_cta);
  cudaError_t err = cudaSuccess;
#define RD_V(VT)                                                                             \
  case VT:                                                                                   \
    err = split ? launch_pdl(8, pre_attn_kernel<KT, VT, true>, grid, block, 0, st, a)        \
                : launch_pdl(8, pre_attn_kernel<KT, VT, false>, grid, block, 0, st, a);      \
    break;
  switch (vt) {
    RD_V(RD_KV_F32)
    RD_V(RD_KV_F16)
    RD_V(RD_KV_Q8_0)
    RD_V(RD_KV_Q4_0)
    RD_V(RD_KV_Q5_0)
    RD_V(RD_KV_Q4_1)
    default: return RD_ERR_TYPE;
  }
#undef RD_V
  return err == cudaSuccess ? RD_OK : RD_ERR_CUDA;
}

int launch_pre_attn(int kt, int vt, const float *qg, const float *k_src, const float *v_src,
                    const float *q_w, const float *k_w, float eps, float *q_out, float *gate_out,
                    void *k_rows, void *v_rows, const int32_t *pos, int n_tok, int n_head, int nkv,
                    int n_rot, float freq_base, cudaStream_t st) {
  if (n_tok == 0) return RD_OK;
  PreAttnArgs a;
  a.qg = qg;
  a.k_src = k_src;
  a.v_src = v_src;
  a.q_w = q_w;
  a.k_w = k_w;
  a.q_out = q_out;
  a.gate_out = gate_out;
  a.k_rows = (uint8_t *)k_rows;
  a.v_rows = (uint8_t *)v_rows;
  a.pos = pos;
  a.n_tok = n_tok;
  a.n_head = n_head;
  a.nkv = nkv;
  a.n_rot = n_rot;
  a.eps = eps;
  a.freq_base = freq_base;
  a.rope = make_rope_table(n_rot, freq_base);
#define RD_K(KT) \
  case KT: return pre_attn_v<KT>(vt, a, st);
  switch (kt) {
    RD_K(RD_KV_F32)
    RD_K(RD_KV_F16)
    RD_K(RD_KV_Q8_0)
    RD_K(RD_KV_Q4_0)
    RD_K(RD_KV_Q5_0)
    RD_K(RD_KV_Q4_1)
    default: return RD_ERR_TYPE;
  }
#undef RD_K
}

}  // namespace rd
