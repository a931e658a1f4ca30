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

// Where the lines lie, measured (us per layer with its pre-attention stage, 4 KV heads: one cluster per KV head /
// step_kernel with records + merge; the two forms of one build):
//   keys       2000         3000         3584         4096         4600         5632         6200         8192
//   f16        10.4 / 11.8  11.3 / 12.7  12.0 / 13.3  12.1 / 13.6  12.7 / 14.0  13.8 / 14.5  15.3 / 14.9  16.6 / 16.3
//   q8_0/f16   10.4 / 11.7  11.6 / 12.5  12.0 / 13.0  12.8 / 13.3  13.4 / 13.5  14.2 / 14.5  15.6 / 14.7  16.9 / 15.7
//   q8_0       10.1 / 11.6  11.5 / 12.4  12.5 / 12.6  12.9 / 12.9  13.5 / 12.9  14.5 / 13.8  15.7 / 14.0  16.8 / 15.5
//   q4_0        9.6 / 11.2  10.4 / 11.7  11.3 / 11.9  11.5 / 12.0  12.1 / 12.1  12.9 / 12.9  14.0 / 12.9  14.8 / 13.8
//   q5_0/q4_1   9.7 / 11.3  10.8 / 12.0  11.7 / 12.3  12.1 / 12.5  12.9 / 12.6  13.8 / 13.3  14.9 / 13.4  16.0 / 14.3
//   q8_0/q4_0   9.9 / 11.3  10.8 / 12.2  12.0 / 12.5  12.4 / 12.6  12.9 / 12.8  13.6 / 13.5  14.8 / 13.6  15.6 / 14.7
// The first line (5632 keys, 3584 for the pairs of three groups) was fitted to slower clusters; today they are the faster
// form, or as fast, up to 4096 keys for those pairs too (0 to 4 % at 4096).
// The second line, and decode_kernel (all heads) before it (step_kernel with records / decode_kernel, merges included):
//   keys       4096         8192         16384        32768        65536
//   f16        12.8 / 18    15.6 / 22    20.8 / 28    32 / 39      -
//   q8_0/f16   12.4 / 16    15.0 / 18    18.7 / 22    28.0 / 30    44.3 / 45.2
//   q8_0       12.0 / 14    14.8 / 17    19.0 / 20    26.1 / 24.8  39.3 / 36.5
//   q4_0       11.8 / 14    13.3 / 16    16.4 / 18    21.4 / 21.9  30.9 / 30.5
// The line at 24576 keys for the other three-group pairs (decode and merge alone, records per head / all heads):
//   keys       4096        16384         24576         32768         65536
//   q5_0/q4_1  8.4 / 11.5  14.2 / 14.8   17.6 / 17.5   20.1 / 19.5   31.3 / 29.1
//   q4_1       7.9 / 11.0  12.7 / 13.9   15.7 / 16.3   17.6 / 17.9   26.1 / 25.6
//   q8_0/q4_0  8.5 / 11.2  14.1 / 14.6   17.0 / 16.6   19.6 / 18.4   31.0 / 27.4
// Fewer KV heads (one cluster per KV head / records per head / all heads). The first line scales with them, which
// keeps clusters a little short of where they stop being faster for one head (8.4 against 8.0 at 4096 keys); the second was
// taken over as it is, although all heads are the slower form there at every length:
//   keys              896               1792              4096              24576          98304
//   2, f16            5.6 / 7.1 / 9.8   7.3 / 7.4 / 9.9   9.4 / 8.2 / 12.5  - / 14.8 / 25  - / 40.1 / 77
//   2, q4_0           5.6 / 7.4 / 9.5   6.4 / 7.5 / 9.5   8.4 / 7.6 / 9.8   - / 11.5 / 15  - / 22.4 / 31
//   2, q5_0/q4_1      5.6 / 7.5 / 9.6   6.4 / 7.6 / 9.7   8.8 / 7.7 / 10.0  - / 12.4 / 16  - / 26.0 / 37
//   1, f16            5.6 / 7.0 / 8.4   7.3 / 7.4 / 8.8   9.2 / 7.9 / 10.2  - / 11.4 / 20  - / 24.1 / 71
//   1, q4_0           5.6 / 7.3 / 9.0   6.1 / 7.6 / 9.0   7.9 / 7.8 / 9.3   - / 9.4 / 14   - / 14.6 / 30
//   1, q5_0/q4_1      5.6 / 7.5 / 9.3   6.2 / 7.9 / 9.3   8.4 / 8.0 / 9.6   - / 10.0 / 15  - / 17.3 / 36
// The cluster form saves the merge launch but uses 64 SMs; records use all. decode_kernel copies all KV heads of
// a key in one box, which costs a long launch fewer issue slots and a short one a larger prologue; with f16
// rows it has shared memory for four or eight warps only.
int step_splits(int kt, int vt, int n_head_kv, int64_t n_keys) {
  const int most = (key_groups(kt, vt) == 1 ? 5632 : 3584) * n_head_kv / 4;
  if (n_keys < 0 || n_keys > most) return 0;
  // at least one slot for some of the warps of each CTA: more CTAs share out the copies, and the
  // latency of a CTA's instruction fetch, down to about two slots each
  return n_keys <= 16 * kSlotKeys ? 8 : 16;
}

int step_record_splits(int kt, int vt, int n_head_kv, int64_t n_keys, int sms) {
  if (n_keys < 0 || (key_groups(kt, vt) == 3 && n_keys > 24576)) return 0;
  return sms / n_head_kv;
}

int decode_tile_keys(int kt, int vt) { return 16 * key_groups(kt, vt); }

}  // namespace rd
