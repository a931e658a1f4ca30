// Internal (C++) launch interface shared by the translation units of the library.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace rd {

struct DeviceStatus;

// ---- rd_kv.cu
int launch_kv_append(int kt, int vt, const float *ks, const float *vs, void *kd, void *vd,
                     int64_t width, int head_dim, int heads_per_tok, const int32_t *pos, int n_rot,
                     float freq_base, cudaStream_t st);
int launch_kv_fill(int type, void *cache, int64_t n_rows, int head_dim, uint32_t seed,
                   cudaStream_t st);
int launch_rope(float *x, int n_tok, int n_heads, int head_dim, int n_rot, float freq_base,
                const int32_t *pos, cudaStream_t st);
int launch_deinterleave(const float *yq, float *q, float *gate, int64_t n_rows, int head_dim,
                        cudaStream_t st);
int launch_sigmoid_gate(float *g, float *y, int64_t n, cudaStream_t st);
// n_values stored values of K (type kt) and V (type vt) -> f16 (the dequantizing loads of
// include/rdna4/kv.h:174-368, rounded once); either with a null source: left out.
struct DequantJob {
  int kt;
  const void *k;
  void *kdst;
  int vt;
  const void *v;
  void *vdst;
  int64_t n_values;
};
int launch_kv_dequant_f16_pair(const DequantJob &job, unsigned *flags, int n_flags, cudaStream_t st);   // zeroes flags, too

// ---- rd_pre.cu
int launch_rms_norm(const float *x, const float *w, float *y, int64_t nrows, int64_t ncols, float eps,
                    cudaStream_t st);
// One launch for deinterleave + q/k RMS-norm + RoPE + K/V quantize-and-store of n_tok
// tokens (head_dim 256, n_rot a multiple of 64).
int launch_pre_attn(int kt, int vt, const float *qg, const float *k_src, const float *v_src,
                    const float *q_w, const float *k_w, float eps, float *q_out, float *gate_out,
                    void *k_rows, void *v_rows, const int32_t *pos, int n_tok, int n_head, int nkv,
                    int n_rot, float freq_base, cudaStream_t st);

// ---- rd_shard.cu (types)
// Exchange buffers of a context-sharded group, as mapped into this process: x[r] is
// rank r's buffer (x[rank] the local one): kShardHeaderBytes of header, then
// [2 parities][world][n_head][4 dim quarters][kXPart] record parts of 8-byte words
// (f32 value, epoch).
constexpr int kShardMaxWorld = 8;
constexpr int kShardMaxHeads = 32;
constexpr int kXPart = 2 + 64;  // (m, l) + one quarter of the accumulator
constexpr size_t kShardHeaderBytes = 256;
struct ShardPeers {
  unsigned char *x[kShardMaxWorld];
  int rank;
  int world;
  unsigned long long wait_ns;  // how long the merge waits for the other ranks' records
};
// ---- rd_decode_*.cu
// One launch of the split-KV decode kernel, one token: attends keys key_begin..(pos ? pos[0] : t), writes
// n_splits records per head into partial[n_head][n_splits][258]. (n_tok > 1: launch_block.)
struct DecodeArgs {
  const float *q;
  const void *k;
  const void *v;
  float *partial;
  const int32_t *pos;  // device, may be null
  int t;
  int key_begin;
  int n_tok;
  int n_head;
  int n_head_kv;
  float scale;
  int n_splits;
  DeviceStatus *status;
  // Fused append (optional, single token only): the f32 rows k_new / v_new
  // [n_head_kv][256] are quantized and stored as cache row `new_row` by the first CTAs of
  // the launch; the keys attended are still key_begin..t (pass t = new_row - 1).
  const float *k_new = nullptr;
  const float *v_new = nullptr;
  int new_row = 0;
  // Context-sharded call (single token): the launch also runs the exchange -- reduces its
  // records per (head, dim quarter), stores the parts into every rank's buffer, waits for
  // the other ranks' parts and writes the merged (optionally gated) output to push_out.
  const ShardPeers *push = nullptr;
  float *push_out = nullptr;    // [n_head][256]
  float *push_gate = nullptr;   // optional
};
int launch_decode(int kt, int vt, const DecodeArgs &a, cudaStream_t st);
// Short contexts, one token (rd_step.cuh): a cluster of n_splits CTAs per KV head attends keys
// key_begin..t and writes the merged, optionally gated output itself (`partial` is not used). With
// k_new / v_new the rows of key t are also quantized and stored as cache row t.
int launch_step(int kt, int vt, const DecodeArgs &a, float *out, float *gate, cudaStream_t st);
// CTAs per KV head of that launch for n_keys keys, or 0 where launch_decode is the faster one (or
// n_keys < 0: not known on the host).
int step_splits(int kt, int vt, int n_head_kv, int64_t n_keys);
// The same kernel with records (out == nullptr: a.n_splits CTAs per KV head write a.partial), for the long
// contexts where that is the faster one: CTAs per KV head, or 0.
int step_record_splits(int kt, int vt, int n_head_kv, int64_t n_keys, int sms);

// Blocks of tokens (rd_block.cuh): token i attends keys 0..pos[i] (on the device); a CTA serves `chunk`
// <= 8 tokens. Writes n_splits records per (token, head) like launch_decode.
int launch_block(int kt, int vt, const DecodeArgs &a, int chunk, cudaStream_t st);
// Tokens per CTA for a block of n_tok: as few chunks as possible, evenly filled.
inline int block_chunk(int n_tok) {
  const int chunks = (n_tok + 7) / 8;
  return (n_tok + chunks - 1) / chunks;
}

// One sequence of a multi-sequence launch, as the kernels read it from device memory.
// The last of the q_len new tokens attends keys 0..t, token i keys 0..t-(q_len-1-i).
// Its records live at records[rec_base ...] as [q_len][n_head][n_splits][258].
struct alignas(64) DecodeSeq {
  alignas(64) unsigned char tm_k[128];  // CUtensorMap over the K cache, if k_tmap
  alignas(64) unsigned char tm_v[128];
  const float *q;    // [q_len][n_head][256]
  const uint8_t *k;
  const uint8_t *v;
  float *out;        // [q_len][n_head][256]
  float *gate;       // optional, like out
  int t;
  int n_splits;
  int rec_base;      // in records
  int k_tmap;
  int v_tmap;
  int pad_;
};
static_assert(sizeof(DecodeSeq) == 320, "DecodeSeq layout");

// launch_decode_multi runs in two phases: with host_seqs set it only encodes the
// tensor maps into the host-side descriptors (k_tmap / v_tmap say which exist); with
// host_seqs null it launches n_items CTAs over the device copies.
struct MultiDecodeArgs {
  DecodeSeq *host_seqs;
  int n_seq;
  const DecodeSeq *dev_seqs;
  const int4 *dev_items;  // (sequence, first token, split, 0)
  int n_items;
  int item_slots;         // 64-key slots of an item, on average, and
  bool waves;             // whether the CTAs are more than a wave (BlockRuns)
  int q_len;
  int n_head;
  int n_head_kv;
  float scale;
  float *records;
  DeviceStatus *status;
};
int launch_decode_multi(int kt, int vt, const MultiDecodeArgs &a, cudaStream_t st);   // q_len 1
int launch_block_multi(int kt, int vt, const MultiDecodeArgs &a, cudaStream_t st);    // q_len > 1
// Keys per tile of the (kt, vt) kernel: the granularity of the key split.
int decode_tile_keys(int kt, int vt);

// ---- rd_tmap.cu
// Tensor map over a KV cache viewed as u64 [n_rows][key bytes / 8] with a box of
// [tile_rows][key bytes / 8 + 2]: one copy brings a whole tile into shared memory with
// a key pitch of key bytes + 16 (the extra columns are outside the tensor: zeros).
// Returns RD_OK, or an error if the key is too wide for one box (f16 / f32 rows), the
// driver entry point is unavailable, or the encoder refuses.
int encode_kv_tmap(void *tmap_out, const void *base, int type, int n_head_kv, int64_t n_rows,
                   int tile_rows);

// Tensor map over an f16 KV cache [n_rows][n_head_kv * 256] with a box of
// [tile_rows][64 dims] and the hardware 128-byte swizzle (what tcgen05.mma descriptors
// with SWIZZLE_128B read).
int encode_f16_tmap(void *tmap_out, const void *base, int n_head_kv, int64_t n_rows, int tile_rows);

// Tensor map over f32 activations [n_rows][n_head][width] with a box of [tokens][heads][32 dims] and the
// hardware 128-byte swizzle.
int encode_f32_tmap(void *tmap_out, const void *base, int width, int n_head, int64_t n_rows, int heads, int tokens);

// ---- rd_prefill.cu
// Causal prefill attention over f16 caches on tcgen05: token i attends keys 0..pos[i]
// (pos on the device), keys_total rows exist in the cache. gate (optional) fuses
// out *= sigmoid(gate); n_rot > 0 applies the partial RoPE to the queries on load.
// splits > 1 (with `records`, prefill_record_bytes(...) bytes): the keys are also split
// over gridDim.z and a second launch merges the per-split records.
struct PrefillPlan {
  int heads;    // of a CTA's rows: 1 (x 128 tokens) or 3 (x 42 tokens)
  int splits;   // of the keys
  int pairs;    // above 0: a balanced launch of that many pairs of CTAs (splits 1)
};
int launch_prefill(const float *q, const void *k, const void *v, float *out, const float *gate,
                   const int32_t *pos, int n_q, int keys_total, int n_head, int n_head_kv, float scale,
                   int n_rot, float freq_base, DeviceStatus *status, float *records, PrefillPlan plan,
                   const float *k_new, const float *v_new, void *k_dst, void *v_dst, bool kv_pending,
                   cudaStream_t st);   // kv_pending: the launch before this one writes k and v, and has waited
                                       // for everything before it (kv_dequant_f16_kernel)
int prefill_splits(int n_q, int keys_total, int n_head, int sms);
size_t prefill_record_bytes(int n_q, int n_head, int splits);
size_t prefill_record_bytes(int n_q, int n_head, PrefillPlan plan);
unsigned *prefill_flags(void *records, PrefillPlan plan);   // 2 pairs words that a launch finds zero, or null
int prefill_tile_tokens(int heads);
int prefill_ctas(PrefillPlan plan, int n_q, int keys_total, int n_head);
PrefillPlan prefill_plan(int n_q, int keys_total, int n_head, int sms, size_t record_bytes);   // with that much memory

// ---- rd_merge.cu
// partial [n_rows][n_splits][258] -> out [n_rows][256]; optional fused sigmoid gate.
int launch_merge(const float *partial, float *out, int n_rows, int n_splits, float *gate,
                 cudaStream_t st);
// The same merge with one more key folded in: the key stored at k_row / v_row (cache row
// of the newest position, types kt / vt, n_head_kv heads) attended by q [n_rows][256]
// with `scale`, as if it were one more record (m = score, l = 1, acc = v). q must not
// alias out.
struct ExtraKey {
  const float *q;
  const uint8_t *k_row;
  const uint8_t *v_row;
  int kt, vt, nkv;
  float scale;
};
int launch_merge_extra(const float *partial, float *out, int n_rows, int n_splits, float *gate,
                       const ExtraKey &x, cudaStream_t st);
// partial [n_rows][n_in][258] -> records [n_rows][n_out][258]: record j merges the
// input records [j*n_in/n_out, (j+1)*n_in/n_out).
int launch_merge_records(const float *partial, float *records, int n_rows, int n_in, int n_out,
                         cudaStream_t st);
// Multi-sequence merge: row (sequence, token, head) reads its n_splits records from the
// sequence's block of `records` and writes (optionally gated) into the sequence's out.
int launch_merge_multi(const DecodeSeq *dev_seqs, const float *records, int n_seq, int q_len,
                       int n_head, int records_per_row, cudaStream_t st);

// Host bytes to the device in kernel parameters (a pageable copy beyond what fits in them): the bytes are
// read during the call. dst 16-byte aligned.
int launch_upload(const void *src, void *dst, size_t bytes, cudaStream_t st);

// ---- rd_shard.cu (launchers)
// partial [n_head][n_in][258] (this rank's split records) -> one record per head stored
// into every rank's buffer, then this call's epoch into every rank's flag.
int launch_shard_push(const float *partial, int n_in, int n_head, const ShardPeers &g,
                      cudaStream_t st);
// Waits (bounded) for all ranks' records of this call, merges them into out
// [n_head][256] (optional fused sigmoid gate) and advances the local epoch.
int launch_shard_merge(float *out, float *gate, int n_head, const ShardPeers &g,
                       DeviceStatus *status, cudaStream_t st);
// Both halves in one launch.
int launch_shard_exchange(const float *partial, int n_in, float *out, float *gate, int n_head,
                          const ShardPeers &g, DeviceStatus *status, cudaStream_t st);

}  // namespace rd
