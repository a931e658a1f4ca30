// Log-sum-exp merge of split-KV partial records (replaces attn_merge_kernel and
// attn_merge_batch_kernel, include/rdna4/attn.cuh:563-590,795-827).
//
//   mm = max_s m_s;  out = sum_s acc_s * e^(m_s - mm) / sum_s l_s * e^(m_s - mm)
//
// A row whose records are all empty (m = -inf) gives zeros, never NaN. The reference
// runs one 32-lane warp per head over at most 16 records; here a head can have one
// record per SM, so a CTA owns (row, 64-dim quarter) and spreads the records over 16
// thread groups: 4 * n_rows CTAs of 1024 threads keep the read of the partial buffer
// wide enough to stay off the critical path of a ~25 us decode step.
#include <string.h>

#include "rd_common.cuh"
#include "rd_internal.h"

namespace rd {

constexpr int kMergeDims = 64;    // dims per CTA
constexpr int kMergeGroups = 16;  // record groups per CTA

// MODE 0: normalised output (optionally gated). MODE 1: un-normalised record out.
// MODE 3: like 0, plus one more key -- the newest position's row, still only in the cache
// -- attended here as one more record (m = scale * q.k, l = 1, acc = v).
template <int MODE>
__global__ void __launch_bounds__(kMergeDims *kMergeGroups, 1)
merge_kernel(const float *__restrict__ partial, float *__restrict__ out, int n_in, int n_out,
             float *__restrict__ gate, const ExtraKey xk) {
  __shared__ float s_l[kMergeGroups];
  __shared__ float s_gm[kMergeGroups];
  __shared__ float s_acc[kMergeGroups][kMergeDims];
  pdl_launch_dependents();
  pdl_wait();

  const int row = blockIdx.x;
  const int quarter = blockIdx.y;
  const int j = MODE == 1 ? blockIdx.z : 0;  // output record index
  const int tx = threadIdx.x % kMergeDims, ty = threadIdx.x / kMergeDims;
  const int lo = MODE == 1 ? (int)(((int64_t)n_in * j) / n_out) : 0;
  const int hi = MODE == 1 ? (int)(((int64_t)n_in * (j + 1)) / n_out) : n_in;
  const float *base = partial + (size_t)row * n_in * kRec;
  // One pass: group ty walks records lo+ty, lo+ty+16, ... and keeps a local log-sum-exp
  // (m, l, acc); the 16 groups are then combined through shared memory. An empty record
  // (m = -inf) weighs nothing and whatever its body holds is never used. The first batch is
  // requested before anything else, the gate value with it. A batch of ten holds the 148 records
  // of a full-GPU decode in ONE round trip to L2 (four per batch took three).
  constexpr int kBatch = 10;
  float mB[kBatch], aB[kBatch], lB[kBatch];
  auto request = [&](int s0) {
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int s = s0 + k * kMergeGroups;
      mB[k] = -INFINITY;
      aB[k] = lB[k] = 0.f;
      if (s < hi) {
        const float *rec = base + (size_t)s * kRec;
        mB[k] = rec[0];
        aB[k] = rec[2 + quarter * kMergeDims + tx];
        if (tx == 0) lB[k] = rec[1];
      }
    }
  };
  request(lo + ty);
  float gate_in = 0.f;
  if (MODE != 1 && gate != nullptr && ty == 0) gate_in = gate[(size_t)row * kHeadDim + quarter * kMergeDims + tx];

  // MODE 3: the score of the extra key, by the first 256 threads (one dim each)
  float x_score = -INFINITY;
  const uint8_t *x_vrow = nullptr;
  if (MODE == 3) {
    __shared__ float s_dot[8];
    const int kvh = row / kGroup;
    float prod = 0.f;
    if (threadIdx.x < kHeadDim)
      prod = xk.q[(size_t)row * kHeadDim + threadIdx.x] *
             load_cache_value(xk.k_row + (size_t)kvh * merge_row_bytes(xk.kt), xk.kt, threadIdx.x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) prod += __shfl_xor_sync(0xffffffffu, prod, o);
    if (threadIdx.x < kHeadDim && (threadIdx.x & 31) == 0) s_dot[threadIdx.x >> 5] = prod;
    __syncthreads();
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) dot += s_dot[i];
    x_score = dot * xk.scale;
    x_vrow = xk.v_row + (size_t)kvh * merge_row_bytes(xk.vt);
  }

  // (its value for this thread's dim: requested here, used after the groups have met)
  float x_val = 0.f;
  if (MODE == 3 && ty == 0) x_val = load_cache_value(x_vrow, xk.vt, quarter * kMergeDims + tx);

  float mloc = -INFINITY, acc = 0.f, ll = 0.f;
  for (int s0 = lo + ty; s0 < hi; s0 += kBatch * kMergeGroups) {
    if (s0 != lo + ty) request(s0);
    float mb = mloc;
#pragma unroll
    for (int k = 0; k < kBatch; ++k) mb = fmaxf(mb, mB[k]);
    if (mb != -INFINITY) {
      const float f = expf(mloc - mb);   // 0 while nothing has been accumulated
      acc *= f;
      ll *= f;
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (mB[k] != -INFINITY) {
          const float w = expf(mB[k] - mb);
          acc = fmaf(aB[k], w, acc);
          ll = fmaf(lB[k], w, ll);
        }
      }
      mloc = mb;
    }
  }
  s_acc[ty][tx] = acc;
  if (tx == 0) {
    s_l[ty] = ll;
    s_gm[ty] = mloc;
  }
  __syncthreads();
  if (ty == 0) {
    float mm = MODE == 3 ? x_score : -INFINITY;
#pragma unroll
    for (int i = 0; i < kMergeGroups; ++i) mm = fmaxf(mm, s_gm[i]);
    float a = 0.f, l = 0.f;
#pragma unroll
    for (int i = 0; i < kMergeGroups; ++i) {
      if (s_gm[i] != -INFINITY) {
        const float w = expf(s_gm[i] - mm);
        a = fmaf(s_acc[i][tx], w, a);
        l = fmaf(s_l[i], w, l);
      }
    }
    const int d = quarter * kMergeDims + tx;
    if (MODE == 3) {
      const float w = expf(x_score - mm);
      a = fmaf(x_val, w, a);
      l += w;
    }
    if (MODE != 1) {
      float o = (mm != -INFINITY && l > 0.f) ? a / l : 0.f;
      float *op = out + (size_t)row * kHeadDim + d;
      if (gate != nullptr) {
        float *gp = gate + (size_t)row * kHeadDim + d;
        const float sg = __fdiv_rn(1.0f, 1.0f + expf(-gate_in));
        *gp = sg;
        o *= sg;
      }
      *op = o;
    } else {
      float *rec = out + ((size_t)row * n_out + j) * kRec;
      rec[2 + d] = a;
      if (d == 0) {
        rec[0] = mm;
        rec[1] = l;
      }
    }
  }
}

// Rows of blocks of tokens and of many sequences: 64 threads of four dims walk a row's records, G such
// groups share a row, a CTA has max(4, G) groups. Bound by the latency of a row's loads, requested eight to
// ten records at a time: G follows the records per row. With a 1024-thread CTA per row and 64 dims, as for the
// 148 records of a long decode, most threads had no record: 64 sequences x 4 tokens x 24 heads took 194
// us, here (G = 1) 14; 120 rows of 37 records 7.6 us, here (G = 4) 5.4, and 4.3 with ten records at a time.
// MULTI: row = (sequence, token, head), records, split count, output and gate from the descriptor.
template <bool MULTI, int G>
__global__ void __launch_bounds__(G > 4 ? 64 * G : 256)
merge_rows_kernel(const float *__restrict__ partial, float *__restrict__ out, int n_rows, int n_in,
                  float *__restrict__ gate, const DecodeSeq *__restrict__ seqs, int rows_per_seq) {
  __shared__ float s_m[G], s_l[G];
  __shared__ float4 s_acc[G][64];
  pdl_launch_dependents();
  pdl_wait();
  const int tx = threadIdx.x & 63, grp = threadIdx.x >> 6;
  const int row = G == 1 ? (int)blockIdx.x * 4 + grp : (int)blockIdx.x;
  if (row >= n_rows) return;   // (G > 1: one row per CTA)
  const float *base = partial + (size_t)row * n_in * kRec;
  int out_row = row;
  if (MULTI) {
    const DecodeSeq &d = seqs[row / rows_per_seq];
    out_row = row % rows_per_seq;
    n_in = d.n_splits;
    base = partial + ((size_t)d.rec_base + (size_t)out_row * n_in) * kRec;
    out = d.out;
    gate = d.gate;
  }
  const size_t at = (size_t)out_row * kHeadDim + 4 * tx;
  const bool last = G == 1 || grp == 0;
  float gv[4] = {0.f, 0.f, 0.f, 0.f};
  if (last && gate != nullptr) {
#pragma unroll
    for (int e = 0; e < 4; ++e) gv[e] = gate[at + e];
  }
  constexpr int kBatch = G == 4 ? 10 : 8;   // (four groups take the 37 records of a quarter of the SMs in one round trip)
  float m = -INFINITY, l = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = G == 1 ? 0 : grp; s0 < n_in; s0 += kBatch * G) {
    float mB[kBatch], lB[kBatch];
    float2 va[kBatch], vb[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int s = s0 + k * G;
      mB[k] = -INFINITY;
      lB[k] = 0.f;
      va[k] = vb[k] = make_float2(0.f, 0.f);
      if (s < n_in) {
        const float *rec = base + (size_t)s * kRec;
        mB[k] = rec[0];
        lB[k] = rec[1];
        va[k] = *reinterpret_cast<const float2 *>(rec + 2 + 4 * tx);   // (a record is 8-byte aligned)
        vb[k] = *reinterpret_cast<const float2 *>(rec + 4 + 4 * tx);
      }
    }
    float mm = m;
#pragma unroll
    for (int k = 0; k < kBatch; ++k) mm = fmaxf(mm, mB[k]);
    if (mm == -INFINITY) continue;
    const float f = expf(m - mm);   // 0 while nothing has been accumulated
    acc.x *= f, acc.y *= f, acc.z *= f, acc.w *= f;
    l *= f;
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      if (mB[k] != -INFINITY) {   // (an empty record weighs nothing, whatever its body holds)
        const float w = expf(mB[k] - mm);
        l = fmaf(lB[k], w, l);
        acc.x = fmaf(va[k].x, w, acc.x);
        acc.y = fmaf(va[k].y, w, acc.y);
        acc.z = fmaf(vb[k].x, w, acc.z);
        acc.w = fmaf(vb[k].y, w, acc.w);
      }
    }
    m = mm;
  }
  if (G > 1) {
    s_acc[grp][tx] = acc;
    if (tx == 0) s_m[grp] = m, s_l[grp] = l;
    __syncthreads();
    if (grp != 0) return;
    float mm = -INFINITY;
#pragma unroll
    for (int i = 0; i < G; ++i) mm = fmaxf(mm, s_m[i]);
    acc = make_float4(0.f, 0.f, 0.f, 0.f);
    l = 0.f;
#pragma unroll
    for (int i = 0; i < G; ++i) {
      if (s_m[i] == -INFINITY) continue;
      const float w = expf(s_m[i] - mm);
      const float4 a = s_acc[i][tx];
      l = fmaf(s_l[i], w, l);
      acc.x = fmaf(a.x, w, acc.x);
      acc.y = fmaf(a.y, w, acc.y);
      acc.z = fmaf(a.z, w, acc.z);
      acc.w = fmaf(a.w, w, acc.w);
    }
    m = mm;
  }
  float o[4] = {0.f, 0.f, 0.f, 0.f};
  if (m != -INFINITY && l > 0.f) o[0] = acc.x / l, o[1] = acc.y / l, o[2] = acc.z / l, o[3] = acc.w / l;
  if (gate != nullptr) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float sg = __fdiv_rn(1.0f, 1.0f + expf(-gv[e]));
      gate[at + e] = sg;
      o[e] *= sg;
    }
  }
  if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    *reinterpret_cast<float4 *>(out + at) = make_float4(o[0], o[1], o[2], o[3]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) out[at + e] = o[e];
  }
}

int launch_merge(const float *partial, float *out, int n_rows, int n_splits, float *gate,
                 cudaStream_t st) {
  if (n_rows == 0) return RD_OK;
  const dim3 grid((unsigned)n_rows, kHeadDim / kMergeDims, 1);
  // up to 64 records: a few hundred rows of a block of tokens, each with 256 threads
  if (n_splits <= 64 && n_rows > 24 && (reinterpret_cast<uintptr_t>(partial) & 7) == 0)
    return launch_pdl(4, merge_rows_kernel<false, 4>, dim3((unsigned)n_rows), dim3(256), 0, st, partial, out, n_rows,
                      n_splits, gate, nullptr, 1) == cudaSuccess
               ? RD_OK
               : RD_ERR_CUDA;
  return launch_pdl(4, merge_kernel<0>, grid, dim3(kMergeDims * kMergeGroups), 0, st, partial, out, n_splits, 1, gate,
                    ExtraKey{}) == cudaSuccess
             ? RD_OK
             : RD_ERR_CUDA;
}

int launch_merge_extra(const float *partial, float *out, int n_rows, int n_splits, float *gate,
                       const ExtraKey &x, cudaStream_t st) {
  if (n_rows == 0) return RD_OK;
  const dim3 grid((unsigned)n_rows, kHeadDim / kMergeDims, 1);
  return launch_pdl(4, merge_kernel<3>, grid, dim3(kMergeDims * kMergeGroups), 0, st, partial, out, n_splits,
                    1, gate, x) == cudaSuccess
             ? RD_OK
             : RD_ERR_CUDA;
}

int launch_merge_records(const float *partial, float *records, int n_rows, int n_in, int n_out,
                         cudaStream_t st) {
  if (n_rows == 0) return RD_OK;
  const dim3 grid((unsigned)n_rows, kHeadDim / kMergeDims, (unsigned)n_out);
  return launch_pdl(4, merge_kernel<1>, grid, dim3(kMergeDims * kMergeGroups), 0, st, partial, records, n_in,
                    n_out, nullptr, ExtraKey{}) == cudaSuccess
             ? RD_OK
             : RD_ERR_CUDA;
}

int launch_merge_multi(const DecodeSeq *dev_seqs, const float *records, int n_seq, int q_len,
                       int n_head, int records_per_row, cudaStream_t st) {
  const int rows = n_seq * q_len * n_head;
  if (rows == 0) return RD_OK;
  // (the average: a row's own count follows its sequence's length)
  const auto kernel = records_per_row <= 12   ? merge_rows_kernel<true, 1>
                      : records_per_row <= 40 ? merge_rows_kernel<true, 4>
                                              : merge_rows_kernel<true, 16>;
  const dim3 grid((unsigned)(records_per_row <= 12 ? (rows + 3) / 4 : rows));
  return launch_pdl(4, kernel, grid, dim3(records_per_row <= 40 ? 256 : 1024), 0, st, records, (float *)nullptr, rows, 0,
                    (float *)nullptr, dev_seqs, q_len * n_head) == cudaSuccess
             ? RD_OK
             : RD_ERR_CUDA;
}

// A copy from pageable memory is a stop for the launches around it (the copy engine, about 5 us); up to 32 KB
// fit into the parameters of a kernel that takes part in the dependent launches.
template <int N>
struct UploadArgs {
  uint4 *dst;
  int n;
  alignas(16) uint4 data[N];
};
template <int N>
__global__ void __launch_bounds__(256) upload_kernel(const __grid_constant__ UploadArgs<N> a) {
  pdl_launch_dependents();
  pdl_wait();
  for (int i = threadIdx.x; i < a.n; i += blockDim.x) a.dst[i] = a.data[i];
}
template <int N>
static int upload(const void *src, void *dst, size_t bytes, cudaStream_t st) {
  static thread_local UploadArgs<N> a;
  a.dst = (uint4 *)dst;
  a.n = (int)((bytes + 15) / 16);
  memcpy(a.data, src, bytes);
  return launch_pdl(4, upload_kernel<N>, dim3(1), dim3(256), 0, st, a) == cudaSuccess ? RD_OK : RD_ERR_CUDA;
}
int launch_upload(const void *src, void *dst, size_t bytes, cudaStream_t st) {
  if (bytes <= 2048) return upload<128>(src, dst, bytes, st);
  if (bytes <= 8192) return upload<512>(src, dst, bytes, st);
  if (bytes <= 32640) return upload<2040>(src, dst, bytes, st);
  return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st) == cudaSuccess ? RD_OK : RD_ERR_CUDA;
}

}  // namespace rd
