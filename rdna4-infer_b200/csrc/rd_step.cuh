// Decode attention of one query token, one KV head per CTA: a cluster per KV head in one launch over
// short contexts, records for merge_kernel over longer ones (step_splits, step_record_splits).
//
// Replaces attn_split_kernel (include/rdna4/attn.cuh:445-560) and the unsplit attn_kernel
// (:95-185). Grid (n_splits, n_head_kv): a CTA owns a contiguous run of 16-key slots of ONE KV
// head and its six query heads. Every warp is on its own: it takes the CTA's slots w, w + W, ...
// and streams them through a private ring with 16-byte asynchronous copies, one commit group per
// slot and tensor, so the key loop has no cross-warp synchronisation at all -- the warp that
// waits, dequantizes and multiplies a slot also re-fills its ring position.
//
// The warps' partial results meet once, in shared memory; then every CTA of the KV head's cluster
// stores each part of its sums into the shared memory of the CTA that owns that part of the output,
// which combines them as soon as all their bytes have arrived and writes the (gated) output: no records,
// no second launch, no remote read.
//
// Copies: a head's row is a narrow piece (144 bytes of q4_0) of a key, and a tensor-map box of
// such rows costs the TMA unit about 13 cycles per row whatever its width: 50 us for the 131001-key
// q4_0 layer where the arithmetic takes 31. Asynchronous 16-byte copies take any row and need no
// descriptor (none to encode on the host).
//
// What bounds it: latency (launch, first slot, the two meetings), with one cluster per KV head from about
// 2000 keys the rate at which 64 SMs can fetch (35 bytes a cycle each). The longest contexts of 4- and 8-bit
// caches go to decode_kernel, whose slots span all KV heads of a key: wide rows for the TMA unit, no copy
// instructions in warps that are bound by the dequantize + mma.sync issue slots (131001 q4_0 keys: 49
// us per layer here, 44 there).
#pragma once
#include "rd_frag.cuh"
#include "rd_internal.h"
#include "rd_quant.cuh"

namespace rd {

// dim table (512), query fragments (3456), new row (2048), received sums (6144) and their (m, l) (768)
constexpr int kStepRecv = 512 + 3456 + 2048;
constexpr int kStepHeader = kStepRecv + 6144 + 768;
constexpr int kMaxCluster = 16;
static_assert(kStepHeader % 16 == 0, "rings are 16-byte aligned");

__host__ __device__ constexpr int step_pair_bytes(int kt, int vt) {
  return kSlotKeys * (slot_pitch(kt) + slot_pitch(vt));
}
// Warps per CTA: as many as have two slots each in the ring budget, up to three per scheduler
// (12 warps leave 168 registers each; the accumulators and query fragments alone are 96).
__host__ __device__ constexpr int step_warps(int kt, int vt) {
  return min_i(12, (kSmemBudget - kStepHeader) / (2 * step_pair_bytes(kt, vt)));
}
template <int KT, int VT>
struct StepGeo {
  static constexpr int kPK = slot_pitch(KT), kPV = slot_pitch(VT);
  static constexpr int kSK = kSlotKeys * kPK, kSV = kSlotKeys * kPV;
  static constexpr int W = step_warps(KT, VT);
  static constexpr int D = min_i(4, (kSmemBudget - kStepHeader) / (W * (kSK + kSV)));
  static constexpr int kSmem = kStepHeader + W * D * (kSK + kSV);
  static_assert(W >= 1 && D >= 1, "ring geometry");
  static_assert(D * (kSK + kSV) >= kGroup * 268 * 4, "a warp's ring holds its epilogue plane");
};

struct StepArgs {
  const float *q;
  const uint8_t *k;
  const uint8_t *v;
  int t;
  int key_begin;
  int nkv;
  float qscale;         // scale * log2(e)
  float *out;
  float *gate;          // optional
  // fused append: the rows of key t, quantized into cache row t by the CTA that attends it
  const float *k_new;
  const float *v_new;
  float *partial;       // records [head][gridDim.x][258] instead of the output, or null
  DeviceStatus *status;
};

__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
// Stores into a CTA of the cluster that complete on its barrier by bytes.
__device__ __forceinline__ void st_async_f32x2(uint32_t a, float x, float y, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(a), "f"(x),
               "f"(y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async_f32x4(uint32_t a, float x, float y, float z, float w, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(a),
               "f"(x), "f"(y), "f"(z), "f"(w), "r"(bar)
               : "memory");
}
// Where a CTA's wait for the others' stores has run out: it stays until no store can reach its shared memory any more,
// that is until every thread of the cluster has ended or has come here, and what those have sent has landed (a
// millisecond is a thousand times what it takes). Every wait in the cluster is bounded, so this one is; whole warps.
__device__ __forceinline__ void cluster_linger() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (const unsigned long long t0 = global_ns(); global_ns() - t0 < 1000000ull;) {}
}
// Softmax reference: p = exp2(s - m) is taken against a reference m that is only moved (and the
// accumulators rescaled) when a score exceeds it by more than kStepSlack, so p <= 2^8 -- exact
// enough in f16 and far from overflow -- and the rescale runs once or twice per warp.
// With one cluster per KV head a warp's runs are longer than those of the all-heads launch, and the weight of the key
// that is the reference is the one that f16 holds exactly: there the reference moves to every slot's own maximum
// (at most kStepSlack below the largest score so far). Error against 64 bits, 4096 f16 keys: 2.76e-4 without, 2.44e-4
// with it, 2.53e-4 in the all-heads launch; 16 layers 194 -> 199 us.
constexpr float kStepSlack = 8.0f;
constexpr float kStepNone = -1.0e30f;   // "no score yet": exp2 of differences needs no special case
constexpr int kPlane = 268;             // floats per head in the epilogue planes (12 mod 32)

template <int KT, int VT>
__global__ void __launch_bounds__(StepGeo<KT, VT>::W * 32, 1)
step_kernel(const __grid_constant__ StepArgs p) {
  using Geo = StepGeo<KT, VT>;
  using KL = KLoad<KT>;
  using VL = VLoad<VT>;
  constexpr int W = Geo::W, D = Geo::D, NT = W * 32, PK = Geo::kPK, PV = Geo::kPV, SK = Geo::kSK, SV = Geo::kSV;
  constexpr int RK = row_bytes(KT), RV = row_bytes(VT);
  constexpr unsigned FULL = 0xffffffffu;

  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float s_m[W][8], s_t[W][8], s_l[W][8];   // per (warp, head): reference, true maximum, sum
  __shared__ float s_wt[W][kGroup];                   // weight of a warp's plane
  __shared__ __align__(8) unsigned long long s_bar;   // the other CTAs' sums
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tq = lane & 3;
  const int kvh = blockIdx.y, nkv = p.nkv;
  const uint32_t sbase = smem_u32(smem);
  unsigned short *inv = reinterpret_cast<unsigned short *>(smem);
  const uint32_t frag0 = sbase + 512;
  uint8_t *stage = smem + 512 + 3456;                 // the appended row: K bytes, then V bytes
  const uint32_t ring_k = sbase + kStepHeader + warp * (D * (SK + SV)), ring_v = ring_k + D * SK;

  // ---- set-up that needs nothing from global memory: dim -> byte offset of the half inside a
  // head's fragment block (inverts KL::dim) ----
  for (int i = threadIdx.x; i < 256; i += NT) {
    const int tq_i = i >> 6, n_i = (i >> 2) & 15, e_i = i & 3;
    inv[KL::dim(tq_i, n_i, e_i)] =
        (unsigned short)(tq_i * kFragPitch + (2 * n_i + (e_i >> 1)) * 4 + (e_i & 1) * 2);
  }
  if (threadIdx.x == 0 && p.partial == nullptr) {
    mbar_init(smem_u32(&s_bar), 1);
    fence_barrier_init();
    mbar_expect_tx(smem_u32(&s_bar), kGroup * kHeadDim * 4 + gridDim.x * kGroup * 8);
  }
  __syncthreads();
  // every CTA of the cluster has started, and its barrier is set up, before another one stores into its shared memory
  // (the matching wait is at the end of the key loop)
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  pdl_wait();   // everything below reads what earlier kernels of the stream wrote

  // the CTA's rank in its cluster, and the cluster's size: a power of two. With records there are no
  // clusters: CTA x of gridDim.x.
  const bool records = p.partial != nullptr;
  const int s = records ? 0 : blockIdx.x, S = records ? 1 : gridDim.x, shift = 31 - __clz(S);
  const int t_last = p.t, key_begin = p.key_begin;
  const bool append = p.k_new != nullptr;
  const int n_keys = t_last >= key_begin ? t_last - key_begin + 1 : 0;
  const int slots_total = (n_keys + kSlotKeys - 1) / kSlotKeys;
  const int c_b = (int)((unsigned)slots_total * blockIdx.x / gridDim.x);   // (below 2^31: 2^22 slots at most)
  const int c_e = (int)((unsigned)slots_total * (blockIdx.x + 1) / gridDim.x);
  const int n_warps = c_e - c_b < W ? c_e - c_b : W;   // warps with slots
  const int n_mine = c_e - c_b > warp ? (c_e - c_b - warp + W - 1) / W : 0;   // slots c_b + warp + it * W
  const int t_load = append ? t_last - 1 : t_last;   // last key that is read from the cache
  const size_t kb = (size_t)nkv * RK, vb = (size_t)nkv * RV;
  const uint8_t *khead = p.k + (size_t)kvh * RK, *vhead = p.v + (size_t)kvh * RV;

  // The query rows of the group: requested before the slots, so that they do not queue behind them.
  constexpr int NQ4 = kGroup * (kHeadDim / 4);   // 384 float4
  constexpr int NQ = (NQ4 + NT - 1) / NT;
  const float4 *q4 = reinterpret_cast<const float4 *>(p.q + (size_t)kvh * kGroup * kHeadDim);
  float4 qv[NQ];
#pragma unroll
  for (int j = 0; j < NQ; ++j)
    if ((int)threadIdx.x + j * NT < NQ4) qv[j] = q4[threadIdx.x + j * NT];

  // ... and so are the values of an appended row, by the CTA that attends it
  const bool owner = append && blockIdx.x == gridDim.x - 1;
  constexpr int NA = (16 + W - 1) / W;   // its 32-value blocks (8 of K, 8 of V) per warp
  float xa[NA];
#pragma unroll
  for (int k = 0; k < NA; ++k) {
    const int b = warp + k * W;
    xa[k] = !owner || b >= 16 ? 0.f
            : b < 8           ? p.k_new[(size_t)kvh * kHeadDim + b * 32 + lane]
                              : p.v_new[(size_t)kvh * kHeadDim + (b - 8) * 32 + lane];
  }

  // The warp's it-th slot into ring position d = it % D; always one commit group, empty behind the end.
  auto fill_k = [&](int it, int d) {
    if (it < n_mine && t_load >= key_begin)
      copy_slot<KT>(ring_k + d * SK, khead, kb, key_begin + (c_b + warp + it * W) * kSlotKeys, t_load, lane);
    cp_async_commit();
  };
  auto fill_v = [&](int it, int d) {
    if (it < n_mine && t_load >= key_begin)
      copy_slot<VT>(ring_v + d * SV, vhead, vb, key_begin + (c_b + warp + it * W) * kSlotKeys, t_load, lane);
    cp_async_commit();
  };
#pragma unroll 1
  for (int it = 0; it < D; ++it) {
    fill_k(it, it);
    fill_v(it, it);
  }
  // Fused append: the CTA that attends key t quantizes its rows of this KV head, one 32-value block
  // per warp, into shared memory; from there into the cache and into the slot that attends them.
  if (owner) {
#pragma unroll
    for (int k = 0; k < NA; ++k) {
      const int b = warp + k * W;
      if (b < 8)
        store_block<KT>(xa[k], stage, b, lane);
      else if (b < 16)
        store_block<VT>(xa[k], stage + RK, b - 8, lane);
    }
  }
  {
    const float qmul = p.qscale * KL::kUnscale;
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
      const int i = threadIdx.x + j * NT;
      if (i < NQ4) {
        const uint32_t hb = frag0 + (uint32_t)(i >> 6) * (4 * kFragPitch);
        const uint2 off = *reinterpret_cast<const uint2 *>(inv + 4 * (i & 63));   // four table entries
        const float x[4] = {qv[j].x, qv[j].y, qv[j].z, qv[j].w};
        const uint32_t o[4] = {off.x & 0xffffu, off.x >> 16, off.y & 0xffffu, off.y >> 16};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const unsigned short hbits = __half_as_ushort(__float2half_rn(x[e] * qmul));
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(hb + o[e]), "h"(hbits) : "memory");
        }
      }
    }
  }
  __syncthreads();
  if (owner) {   // the appended rows into the cache, 4 bytes at a time
    uint32_t *kd = reinterpret_cast<uint32_t *>(const_cast<uint8_t *>(khead) + (size_t)t_last * kb);
    uint32_t *vd = reinterpret_cast<uint32_t *>(const_cast<uint8_t *>(vhead) + (size_t)t_last * vb);
    const uint32_t *st = reinterpret_cast<const uint32_t *>(stage);
    for (int i = threadIdx.x; i < (RK + RV) / 4; i += NT) (i < RK / 4 ? kd[i] : vd[i - RK / 4]) = st[i];
  }
  // the appended row into the slot; the rows behind it are zeros, by the slot's copy or, where nothing was
  // copied, from here
  auto patch = [&](uint32_t slot, int pitch, const uint8_t *row, int words, int row0) {
    const int first = t_last - row0, last = t_load < key_begin ? kSlotKeys - 1 : first;
#pragma unroll 1
    for (int r = first; r <= last; ++r)
#pragma unroll 4
      for (int c = lane; c < words; c += 32)
        *reinterpret_cast<uint32_t *>(smem + (slot - sbase) + r * pitch + 4 * c) =
            r == first ? reinterpret_cast<const uint32_t *>(row)[c] : 0u;
    __syncwarp();
  };

  // ---- key loop ----
  float O[16][4];
  float m0 = kStepNone, m1 = kStepNone;       // softmax references of the lane's two head columns
  float run0 = kStepNone, run1 = kStepNone;   // lane-local true maxima
  float l0 = 0.f, l1 = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) O[i][0] = O[i][1] = O[i][2] = O[i][3] = 0.f;
  // Q fragments (B operand): lane (g, tq) holds head g's 32 words; padding heads are 0.
  uint32_t qb[16][2];
  {
    const uint32_t fa = frag0 + (uint32_t)((g < kGroup ? g : 0) * 4 + tq) * kFragPitch;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint4 v = lds128(fa + 16 * i);
      qb[2 * i][0] = g < kGroup ? v.x : 0u;
      qb[2 * i][1] = g < kGroup ? v.y : 0u;
      qb[2 * i + 1][0] = g < kGroup ? v.z : 0u;
      qb[2 * i + 1][1] = g < kGroup ? v.w : 0u;
    }
  }
  int d = 0;   // ring position of the next slot
#pragma unroll 1
  for (int it = 0; it < n_mine; ++it) {
    const int row0 = key_begin + (c_b + warp + it * W) * kSlotKeys;
    const bool tail = row0 + kSlotKeys - 1 >= t_last;   // ends at or behind the last key
    const uint32_t kslot = ring_k + d * SK, vslot = ring_v + d * SV;
    // groups are committed in the order K0 V0 K1 V1 ...: 2 D - 1 younger ones may be in flight
    cp_async_wait<2 * D - 1>();
    __syncwarp();
    if (owner && tail) patch(kslot, PK, stage, RK / 4, row0);
    // ---- S = K Q^T (16 keys x 8 heads), two accumulator chains ----
    float Sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    KL::run(kslot + g * PK, kslot + (g + 8) * PK, tq, [&](int n, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
      mma16816(Sc[n & 1], a0, a1, a2, a3, qb[n][0], qb[n][1]);
    });
    __syncwarp();
    fill_k(it + D, d);
    float Sv[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) Sv[e] = Sc[0][e] + Sc[1][e];
    if (tail) {   // keys behind the last attended one
      if (row0 + g > t_last) Sv[0] = Sv[1] = -INFINITY;
      if (row0 + g + 8 > t_last) Sv[2] = Sv[3] = -INFINITY;
    }
    const float x0 = fmaxf(Sv[0], Sv[2]), x1 = fmaxf(Sv[1], Sv[3]);
    run0 = fmaxf(run0, x0);
    run1 = fmaxf(run1, x1);
    // ---- online softmax (per head: columns 2t and 2t+1 of this lane) ----
    if (!records || __any_sync(FULL, run0 > m0 + kStepSlack || run1 > m1 + kStepSlack)) {
      // move the references to the maxima of the columns (over the 8 row lanes): of the slot, or of all so far
      float n0 = records ? run0 : x0, n1 = records ? run1 : x1;
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        n0 = fmaxf(n0, __shfl_xor_sync(FULL, n0, o));
        n1 = fmaxf(n1, __shfl_xor_sync(FULL, n1, o));
      }
      if (records) {
        n0 = fmaxf(n0, m0);
        n1 = fmaxf(n1, m1);
      } else {
        run0 = fmaxf(run0, n0);
        run1 = fmaxf(run1, n1);
        n0 = fmaxf(n0, run0 - kStepSlack);
        n1 = fmaxf(n1, run1 - kStepSlack);
      }
      const float c0 = ex2(m0 - n0), c1 = ex2(m1 - n1);
      m0 = n0;
      m1 = n1;
      l0 *= c0;
      l1 *= c1;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        O[j][0] *= c0;
        O[j][1] *= c1;
        O[j][2] *= c0;
        O[j][3] *= c1;
      }
    }
    const float p0 = ex2(Sv[0] - m0), p1 = ex2(Sv[1] - m1), p2 = ex2(Sv[2] - m0), p3 = ex2(Sv[3] - m1);
    l0 += p0 + p2;
    l1 += p1 + p3;
    // P^T fragments: (keys 2t,2t+1 | head g) and (keys 2t+8,2t+9 | head g)
    const uint32_t pb0 = movmatrix_trans(pack_h2(p0, p1)), pb1 = movmatrix_trans(pack_h2(p2, p3));
    // ---- O^T += V^T P^T (256 dims x 8 heads) ----
    cp_async_wait<2 * D - 1>();
    __syncwarp();
    if (owner && tail) patch(vslot, PV, stage + RK, RV / 4, row0);
    const uint32_t r0 = vslot + (uint32_t)(2 * tq) * PV;
    const uint32_t rows[4] = {r0, r0 + PV, r0 + 8 * PV, r0 + 9 * PV};
    VL::run(rows, g, [&](int m, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
      mma16816(O[m], a0, a1, a2, a3, pb0, pb1);
    });
    __syncwarp();
    fill_v(it + D, d);
    if (++d == D) d = 0;
  }
  cp_async_wait<0>();   // (only empty groups are left)
  // ---- the warps meet: sums and maxima over the 8 key-row lanes of each head column, the
  // accumulators (relative to this warp's references) into a plane [head][dim] over its own ring ----
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    l0 += __shfl_xor_sync(FULL, l0, o);
    l1 += __shfl_xor_sync(FULL, l1, o);
    run0 = fmaxf(run0, __shfl_xor_sync(FULL, run0, o));
    run1 = fmaxf(run1, __shfl_xor_sync(FULL, run1, o));
  }
  if (g == 0) {
    s_m[warp][2 * tq] = m0, s_m[warp][2 * tq + 1] = m1;
    s_t[warp][2 * tq] = run0, s_t[warp][2 * tq + 1] = run1;
    s_l[warp][2 * tq] = l0, s_l[warp][2 * tq + 1] = l1;
  }
  constexpr uint32_t kPlaneStride = D * (SK + SV);
  if (tq < kGroup / 2) {
    // Dim d of a head sits at 33 * (d >> 5) + (d & 31) and heads are kPlane floats apart, which
    // spreads the 8 row lanes (32 dims apart for the block loaders) and the quad lanes over banks.
    float *plane = reinterpret_cast<float *>(smem + kStepHeader + warp * kPlaneStride) + 2 * tq * kPlane;
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int d0 = VL::dim(g, m, 0), d1 = VL::dim(g, m, 1);
      const int a0 = 33 * (d0 >> 5) + (d0 & 31), a1 = 33 * (d1 >> 5) + (d1 & 31);
      plane[a0] = O[m][0];
      plane[a0 + kPlane] = O[m][1];
      plane[a1] = O[m][2];
      plane[a1 + kPlane] = O[m][3];
    }
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  __syncthreads();
  // A head per warp, the CTA's warps over its lanes: the CTA's maximum and sum, and the weights of the warps' planes.
  // (references never exceed the true maximum)
  auto combine = [&](auto &&emit) {
    for (int h = warp; h < kGroup; h += W) {
      const bool on = lane < n_warps;
      float mm = on ? s_t[lane][h] : kStepNone;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(FULL, mm, o));
      mm = __shfl_sync(FULL, mm, 0);
      const float w = on ? ex2(s_m[lane][h] - mm) : 0.f;
      float ll = on ? s_l[lane][h] * w : 0.f;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) ll += __shfl_xor_sync(FULL, ll, o);
      ll = __shfl_sync(FULL, ll, 0);
      if (lane < W) s_wt[lane][h] = w * VL::kUnscale;
      emit(h, mm, ll);
    }
  };
  if (records) {   // a CTA's record per head, for merge_kernel
    __shared__ float s_ml[kGroup][2];
    combine([&](int h, float mm, float ll) {
      if (lane == 0) {
        s_ml[h][0] = mm > 0.5f * kStepNone ? mm * 0.6931471805599453f : -INFINITY;   // natural log
        s_ml[h][1] = mm > 0.5f * kStepNone ? ll : 0.f;
      }
    });
    __syncthreads();
    for (int i = threadIdx.x; i < kGroup * (kHeadDim / 4); i += NT) {
      const int h = i >> 6, dd = 4 * (i & 63);
      const int off = h * kPlane + 33 * (dd >> 5) + (dd & 31);
      float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
      for (int w = 0; w < n_warps; ++w) {
        const float *pl = reinterpret_cast<const float *>(smem + kStepHeader + w * kPlaneStride) + off;
        const float wt = s_wt[w][h];
#pragma unroll
        for (int e = 0; e < 4; ++e) a[e] = fmaf(pl[e], wt, a[e]);
      }
      float *rec = p.partial + ((size_t)(kvh * kGroup + h) * gridDim.x + blockIdx.x) * kRec;
      if (dd == 0) rec[0] = s_ml[h][0], rec[1] = s_ml[h][1];
      *reinterpret_cast<float2 *>(rec + 2 + dd) = make_float2(a[0], a[1]);
      *reinterpret_cast<float2 *>(rec + 4 + dd) = make_float2(a[2], a[3]);
    }
    return;
  }
  const uint32_t recv = sbase + kStepRecv, recv_ml = recv + 6144;   // [src][1536 / S] and [src][head][2]
  const uint32_t bar = smem_u32(&s_bar);
  combine([&](int h, float mm, float ll) {   // to every CTA
    if (lane < S) st_async_f32x2(peer_addr(recv_ml + 8 * (s * kGroup + h), lane), mm, ll, peer_addr(bar, lane));
  });
  __syncthreads();
  const int part = kGroup * kHeadDim >> shift;   // output values per CTA: a multiple of 32
  for (int i = threadIdx.x; i < kGroup * (kHeadDim / 4); i += NT) {
    const int h = i >> 6, dd = 4 * (i & 63);
    const int off = h * kPlane + 33 * (dd >> 5) + (dd & 31);
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int w = 0; w < n_warps; ++w) {
      const float *pl = reinterpret_cast<const float *>(smem + kStepHeader + w * kPlaneStride) + off;
      const float wt = s_wt[w][h];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = fmaf(pl[e], wt, a[e]);
    }
    const int owner_rank = 4 * i / part, at = 4 * i - owner_rank * part;
    st_async_f32x4(peer_addr(recv + 4 * (s * part + at), owner_rank), a[0], a[1], a[2], a[3], peer_addr(bar, owner_rank));
  }
  const int e = s * part + threadIdx.x;   // this CTA's part of the output: at most NQ passes
  float gate_in = 0.f;
  if (p.gate != nullptr && (int)threadIdx.x < part) gate_in = p.gate[(size_t)kvh * kGroup * kHeadDim + e];
  // Every CTA waits for its own parts only, by bytes. (With a barrier of the whole cluster and the
  // release of every thread's stores before it, and the combinations above thread by thread over all warps, the kernel
  // spent 5700 of its 9300 cycles behind the key loop: 137 f16 keys 8.11 us a layer, now 7.46, 4096 12.41 and 11.47.)
  const bool ok = mbar_wait(bar, 0, p.status, 40);
  for (int i = threadIdx.x; i < part; i += NT) {   // (whole warps, each within one head)
    const int el = s * part + i, h = el >> 8;
    const size_t at = (size_t)kvh * kGroup * kHeadDim + el;
    if (i != (int)threadIdx.x && p.gate != nullptr) gate_in = p.gate[at];
    // the sources' maxima and sums over the lanes
    const float2 ml = lane < S ? reinterpret_cast<const float2 *>(smem + kStepRecv + 6144)[lane * kGroup + h]
                               : make_float2(kStepNone, 0.f);
    const float *a = reinterpret_cast<const float *>(smem + kStepRecv) + i;
    float mm = ml.x;
#pragma unroll
    for (int o2 = 8; o2 > 0; o2 >>= 1) mm = fmaxf(mm, __shfl_xor_sync(FULL, mm, o2));
    mm = __shfl_sync(FULL, mm, 0);
    const float w = lane < S ? ex2(ml.x - mm) : 0.f;
    float l = ml.y * w, o = 0.f;
#pragma unroll
    for (int o2 = 8; o2 > 0; o2 >>= 1) l += __shfl_xor_sync(FULL, l, o2);
    l = __shfl_sync(FULL, l, 0);
#pragma unroll 4
    for (int c = 0; c < S; ++c) o = fmaf(a[c * part], __shfl_sync(FULL, w, c), o);
    o = ok && mm > 0.5f * kStepNone && l > 0.f ? o / l : 0.f;
    if (p.gate != nullptr) {
      const float sg = __fdiv_rn(1.0f, 1.0f + expf(-gate_in));
      p.gate[at] = sg;
      o *= sg;
    }
    p.out[at] = o;
  }
  if (!__all_sync(FULL, ok)) cluster_linger();
}

// Grid (n_splits, n_head_kv), a cluster per KV head.
template <int KT, int VT>
int launch_step_typed(const DecodeArgs &a, float *out, float *gate, cudaStream_t st) {
  using Geo = StepGeo<KT, VT>;
  static bool attr_set[32] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return RD_ERR_CUDA;
  if (dev < 0 || dev >= 32 || !attr_set[dev]) {
    if (cudaFuncSetAttribute(step_kernel<KT, VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo::kSmem) !=
        cudaSuccess)
      return RD_ERR_CUDA;
    // clusters of 16 are beyond the portable size
    if (cudaFuncSetAttribute(step_kernel<KT, VT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
      return RD_ERR_CUDA;
    if (dev >= 0 && dev < 32) attr_set[dev] = true;
  }
  StepArgs k;
  k.q = a.q;
  k.k = (const uint8_t *)a.k;
  k.v = (const uint8_t *)a.v;
  k.t = a.t;
  k.key_begin = a.key_begin;
  k.nkv = a.n_head_kv;
  k.qscale = a.scale * 1.4426950408889634f;
  k.out = out;
  k.gate = gate;
  k.k_new = a.k_new;
  k.v_new = a.v_new;
  k.partial = out == nullptr ? a.partial : nullptr;
  k.status = a.status;
  return launch_pdl_cluster(step_kernel<KT, VT>, dim3((unsigned)a.n_splits, (unsigned)a.n_head_kv),
                            dim3(Geo::W * 32), Geo::kSmem, out == nullptr ? 1u : (unsigned)a.n_splits, st, k) == cudaSuccess
             ? RD_OK
             : RD_ERR_CUDA;
}

}  // namespace rd
