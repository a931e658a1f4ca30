// A CTA whose wait for a peer's store has run out stays until the store has landed (cluster_linger, rd_step.cuh): a
// cluster of two, CTA 1 stores 20 ms after CTA 0 has given up after 1 ms. Prints "gave up G, value V".
#include <cstdio>

#include "rd_step.cuh"

namespace rd {

__global__ void __cluster_dims__(2, 1, 1) late_store(int *gave_up, float *value) {
  __shared__ float s_value[2];
  __shared__ __align__(8) unsigned long long s_bar;
  const uint32_t bar = smem_u32(&s_bar), at = smem_u32(s_value);
  if (threadIdx.x == 0) {
    s_value[0] = s_value[1] = 0.f;
    mbar_init(bar, 1);
    fence_barrier_init();
    mbar_expect_tx(bar, 8);
  }
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  const unsigned long long t0 = global_ns();
  if (blockIdx.x == 1) {
    while (global_ns() - t0 < 20000000ull) {}
    if (threadIdx.x == 0) st_async_f32x2(peer_addr(at, 0), 1.f, 42.f, peer_addr(bar, 0));
    return;
  }
  bool ok = false;
  while (!ok && global_ns() - t0 < 1000000ull) ok = mbar_test_wait(bar, 0);
  if (!__all_sync(0xffffffffu, ok)) cluster_linger();
  if (threadIdx.x == 0) {
    *gave_up = !ok;
    *value = mbar_test_wait(bar, 0) ? s_value[1] : -1.f;
  }
}

}  // namespace rd

int main() {
  int *g, gave_up = -1;
  float *v, value = -1.f;
  if (cudaMalloc(&g, 4) != cudaSuccess || cudaMalloc(&v, 4) != cudaSuccess) return 1;
  rd::late_store<<<2, 64>>>(g, v);
  if (cudaDeviceSynchronize() != cudaSuccess) return 2;
  cudaMemcpy(&gave_up, g, 4, cudaMemcpyDeviceToHost);
  cudaMemcpy(&value, v, 4, cudaMemcpyDeviceToHost);
  std::printf("gave up %d, value %g\n", gave_up, value);
  return 0;
}
