// Type dispatch of the decode-side attention kernels (instantiations live in rd_decode_k_*.cu and
// rd_block_k_*.cu so that they compile in parallel).
#include "rd_common.cuh"
#include "rd_internal.h"
#include "rd_step.cuh"

namespace rd {

int launch_decode_k_f32(int vt, const DecodeArgs &a, cudaStream_t st);
int launch_decode_k_f16(int vt, const DecodeArgs &a, cudaStream_t st);
int launch_decode_k_q8_0(int vt, const DecodeArgs &a, cudaStream_t st);
int launch_decode_k_q4_0(int vt, const DecodeArgs &a, cudaStream_t st);
int launch_decode_k_q5_0(int vt, const DecodeArgs &a, cudaStream_t st);
int launch_decode_k_q4_1(int vt, const DecodeArgs &a, cudaStream_t st);

int launch_decode_multi_k_f32(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_decode_multi_k_f16(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_decode_multi_k_q8_0(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_decode_multi_k_q4_0(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_decode_multi_k_q5_0(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_decode_multi_k_q4_1(int vt, const MultiDecodeArgs &a, cudaStream_t st);

int launch_decode_multi(int kt, int vt, const MultiDecodeArgs &a, cudaStream_t st) {
  switch (kt) {
    case RD_KV_F32: return launch_decode_multi_k_f32(vt, a, st);
    case RD_KV_F16: return launch_decode_multi_k_f16(vt, a, st);
    case RD_KV_Q8_0: return launch_decode_multi_k_q8_0(vt, a, st);
    case RD_KV_Q4_0: return launch_decode_multi_k_q4_0(vt, a, st);
    case RD_KV_Q5_0: return launch_decode_multi_k_q5_0(vt, a, st);
    case RD_KV_Q4_1: return launch_decode_multi_k_q4_1(vt, a, st);
    default: return RD_ERR_UNSUPPORTED;
  }
}

int launch_decode(int kt, int vt, const DecodeArgs &a, cudaStream_t st) {
  switch (kt) {
    case RD_KV_F32: return launch_decode_k_f32(vt, a, st);
    case RD_KV_F16: return launch_decode_k_f16(vt, a, st);
    case RD_KV_Q8_0: return launch_decode_k_q8_0(vt, a, st);
    case RD_KV_Q4_0: return launch_decode_k_q4_0(vt, a, st);
    case RD_KV_Q5_0: return launch_decode_k_q5_0(vt, a, st);
    case RD_KV_Q4_1: return launch_decode_k_q4_1(vt, a, st);
    default: return RD_ERR_UNSUPPORTED;
  }
}

int launch_step_k_f32(int vt, const DecodeArgs &a, float *out, float *gate, cudaStream_t st);
int launch_step_k_f16(int vt, const DecodeArgs &a, float *out, float *gate, cudaStream_t st);
int launch_step_k_q8_0(int vt, const DecodeArgs &a, float *out, float *gate, cudaStream_t st);
int launch_step_k_q4_0(int vt, const DecodeArgs &a, float *out, float *gate, cudaStream_t st);
int launch_step_k_q5_0(int vt, const DecodeArgs &a, float *out, float *gate, cudaStream_t st);
int launch_step_k_q4_1(int vt, const DecodeArgs &a, float *out, float *gate, cudaStream_t st);

int launch_step(int kt, int vt, const DecodeArgs &a, float *out, float *gate, cudaStream_t st) {
  switch (kt) {
    case RD_KV_F32: return launch_step_k_f32(vt, a, out, gate, st);
    case RD_KV_F16: return launch_step_k_f16(vt, a, out, gate, st);
    case RD_KV_Q8_0: return launch_step_k_q8_0(vt, a, out, gate, st);
    case RD_KV_Q4_0: return launch_step_k_q4_0(vt, a, out, gate, st);
    case RD_KV_Q5_0: return launch_step_k_q5_0(vt, a, out, gate, st);
    case RD_KV_Q4_1: return launch_step_k_q4_1(vt, a, out, gate, st);
    default: return RD_ERR_UNSUPPORTED;
  }
}

int launch_block_k_f32(int vt, const DecodeArgs &a, int chunk, cudaStream_t st);
int launch_block_k_f16(int vt, const DecodeArgs &a, int chunk, cudaStream_t st);
int launch_block_k_q8_0(int vt, const DecodeArgs &a, int chunk, cudaStream_t st);
int launch_block_k_q4_0(int vt, const DecodeArgs &a, int chunk, cudaStream_t st);
int launch_block_k_q5_0(int vt, const DecodeArgs &a, int chunk, cudaStream_t st);
int launch_block_k_q4_1(int vt, const DecodeArgs &a, int chunk, cudaStream_t st);

int launch_block(int kt, int vt, const DecodeArgs &a, int chunk, cudaStream_t st) {
  switch (kt) {
    case RD_KV_F32: return launch_block_k_f32(vt, a, chunk, st);
    case RD_KV_F16: return launch_block_k_f16(vt, a, chunk, st);
    case RD_KV_Q8_0: return launch_block_k_q8_0(vt, a, chunk, st);
    case RD_KV_Q4_0: return launch_block_k_q4_0(vt, a, chunk, st);
    case RD_KV_Q5_0: return launch_block_k_q5_0(vt, a, chunk, st);
    case RD_KV_Q4_1: return launch_block_k_q4_1(vt, a, chunk, st);
    default: return RD_ERR_UNSUPPORTED;
  }
}

int launch_block_multi_k_f32(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_block_multi_k_f16(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_block_multi_k_q8_0(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_block_multi_k_q4_0(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_block_multi_k_q5_0(int vt, const MultiDecodeArgs &a, cudaStream_t st);
int launch_block_multi_k_q4_1(int vt, const MultiDecodeArgs &a, cudaStream_t st);

int launch_block_multi(int kt, int vt, const MultiDecodeArgs &a, cudaStream_t st) {
  switch (kt) {
    case RD_KV_F32: return launch_block_multi_k_f32(vt, a, st);
    case RD_KV_F16: return launch_block_multi_k_f16(vt, a, st);
    case RD_KV_Q8_0: return launch_block_multi_k_q8_0(vt, a, st);
    case RD_KV_Q4_0: return launch_block_multi_k_q4_0(vt, a, st);
    case RD_KV_Q5_0: return launch_block_multi_k_q5_0(vt, a, st);
    case RD_KV_Q4_1: return launch_block_multi_k_q4_1(vt, a, st);
    default: return RD_ERR_UNSUPPORTED;
  }
}

// Where the line lies, measured (us per layer with its pre-attention stage, 4 KV heads, this kernel /
// decode_kernel + merge): q8_0 4096 keys 12.9 / 14.5, 8192 16.7 / 16.9, 12288 20.8 / 18.7; q4_0 8192 14.6 /
// 15.8, 12288 17.3 / 16.7; q8_0/f16 12288 19.7 / 19.9; f16 16384 22.8 / 27.6. 64 SMs fetch a long context
// more slowly than 148, and the wider the rows the later that shows, as decode_kernel has fewer warps
// then (key_groups). With fewer KV heads fewer SMs work here, not there.
int step_splits(int kt, int vt, int n_head_kv, int64_t n_keys) {
  const int groups = key_groups(kt, vt);
  int64_t most = groups == 3 ? 8192 : groups == 2 ? 12288 : 24576;
  if (n_head_kv < 4 && most > 6144) most = 6144;
  if (n_keys < 0 || n_keys > most) return 0;
  // at least one slot for some of the warps of each CTA: more CTAs share out the copies, and the
  // latency of a CTA's instruction fetch, down to about two slots each
  return n_keys <= 16 * kSlotKeys ? 8 : 16;
}

int step_record_splits(int kt, int vt, int n_head_kv, int64_t n_keys, int sms) {
  if (n_keys < 0 || key_groups(kt, vt) > 1) return 0;
  return sms / n_head_kv;
}

int decode_tile_keys(int kt, int vt) { return 16 * key_groups(kt, vt); }

}  // namespace rd
