// Token-block attention kernels whose K cache is f32, one instantiation per V type.
#include "rd_block.cuh"

namespace rd {
int launch_block_k_f32(int vt, const DecodeArgs &a, int chunk, cudaStream_t st) {
  switch (vt) {
    case RD_KV_F32: return launch_block_typed<RD_KV_F32, RD_KV_F32>(a, chunk, st);
    case RD_KV_F16: return launch_block_typed<RD_KV_F32, RD_KV_F16>(a, chunk, st);
    case RD_KV_Q8_0: return launch_block_typed<RD_KV_F32, RD_KV_Q8_0>(a, chunk, st);
    case RD_KV_Q4_0: return launch_block_typed<RD_KV_F32, RD_KV_Q4_0>(a, chunk, st);
    case RD_KV_Q5_0: return launch_block_typed<RD_KV_F32, RD_KV_Q5_0>(a, chunk, st);
    case RD_KV_Q4_1: return launch_block_typed<RD_KV_F32, RD_KV_Q4_1>(a, chunk, st);
    default: return RD_ERR_UNSUPPORTED;
  }
}
int launch_block_multi_k_f32(int vt, const MultiDecodeArgs &a, cudaStream_t st) {
  switch (vt) {
    case RD_KV_F32: return launch_block_multi_typed<RD_KV_F32, RD_KV_F32>(a, st);
    case RD_KV_F16: return launch_block_multi_typed<RD_KV_F32, RD_KV_F16>(a, st);
    case RD_KV_Q8_0: return launch_block_multi_typed<RD_KV_F32, RD_KV_Q8_0>(a, st);
    case RD_KV_Q4_0: return launch_block_multi_typed<RD_KV_F32, RD_KV_Q4_0>(a, st);
    case RD_KV_Q5_0: return launch_block_multi_typed<RD_KV_F32, RD_KV_Q5_0>(a, st);
    case RD_KV_Q4_1: return launch_block_multi_typed<RD_KV_F32, RD_KV_Q4_1>(a, st);
    default: return RD_ERR_UNSUPPORTED;
  }
}
}  // namespace rd
