// Causal prefill attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA).
//
// Replaces attn_fa2_prefill_kernel (include/rdna4/attn_fa2.cuh:30-169 of the reference)
// for f16 K/V caches. One CTA owns a tile of 128 query tokens of ONE query head and walks
// the keys in tiles of 128, in a pair (cta_group::2) with the CTA of the KV head's next query head:
// each loads half of every K and V tile and the pair's MMAs (M = 256, issued by the leader) read
// both halves. Alone, a CTA moves 320 KB through shared memory per tile (operands 192, copies
// 128), 2500 cycles at 128 bytes a cycle against 2048 of tensor-core work; in a pair 192 KB. Tensor memory (512 columns x 128 lanes, lane = query row):
//   columns   0..255  O, the f32 output accumulator
//   columns 256..383  the f32 scores of one tile: the next tile's can be computed as soon as
//                     the softmax warps have these in registers
//   columns 384..511  two buffers of 64 columns for the f16 P of a tile (the A operand of
//                     O += P V, read from TMEM)
// Shared memory (224 KB): Q as f16 in the K-major 128-byte-swizzled layout (64 KB), a ring
// of three half K tiles (96 KB) and a ring of two half V tiles (64 KB), filled by TMA with the
// hardware 128B swizzle.
//
//   prologue   the 128 x 256 f32 query rows -> optional partial RoPE, scale*log2(e), f16,
//              swizzled into shared memory;
//   per 128-key tile j:
//     warp 9     S = Q K_j^T        16 x tcgen05.mma M256 N128 K16
//     warps 0-7  one thread per query row and tile parity (warps 0-3 the even tiles, 4-7 the odd ones),
//                all 128 scores of the row in its registers, the reference maximum handed from tile to
//                tile through shared memory: tcgen05.ld the scores, causal mask (key <= pos[r]), LAZY
//                rescale (the reference point only moves when a row's max grows by more than 2^8, so
//                P stays below 256 in f16 and O in TMEM is rarely touched), P -> f16 pairs, tcgen05.st
//                O += P V_j-2        8 x tcgen05.mma M256 N256 K16 (A = P from TMEM, B = V
//                                   MN-major)
//   epilogue   O / l (times sigmoid(gate) if asked) through shared memory to TMA stores.
// Warps 8 and 10 are the K and V TMA producers (separate warps: a lane parked in
// mbarrier.try_wait parks its whole warp).
//
// What orders the tiles: S of tile j + 1 waits for the LOADS of tile j's scores only, P of tile j for
// P V of tile j - 2. (With P written over its own scores, S of tile j + 2 waited for P V of tile j, a chain
// S - softmax - P V - S of 6300 cycles per two tiles against 4096 of tensor-core work.) A tile takes 2060
// cycles, the tensor core's own rate.
//
// Synchronisation is mbarriers only (TMA transaction counts, tcgen05.commit); every wait
// is bounded and a timeout unwinds the pair (TMEM is always freed). No multicast loads.
#include <stdlib.h>
#include <string.h>

#include <algorithm>

#include "rd_common.cuh"
#include "rd_internal.h"
#include "rd_tc.cuh"

// Timing experiments (skip one pipeline stage, bit mask in PrefillArgs::debug) exist only
// in builds with -DRD_TIMING_SWITCHES; a default build compiles them out.
#ifdef RD_TIMING_SWITCHES
#define RD_PF_DEBUG(p) ((p).debug)
#else
#define RD_PF_DEBUG(p) 0
#endif
// -DRD_PF_TRACING (timing builds only): phase trace of CTA (0, 0, 0),
// [role 0..3][tile 0..47][point 0..7] clock64 values, read back with rd_debug_pf_trace
#ifdef RD_PF_TRACING
__device__ unsigned long long g_pf_trace[4][48][8];
#define RD_PF_TRACE(role, j, pt)                                                  \
  do {                                                                            \
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && (j) < 48)        \
      g_pf_trace[role][j][pt] = clock64();                                        \
  } while (0)
#else
#define RD_PF_TRACE(role, j, pt) do { } while (0)
#endif

namespace rd {

constexpr int kPfM = 128;                 // query rows per CTA
constexpr int kPfN = 128;                 // keys per tile
constexpr int kPfQBytes = kPfM * kHeadDim * 2;             // 65536 (also the epilogue staging)
// A CTA of the pair holds half of each K tile (64 of the 128 keys) and of each V tile (128 of the 256 dims).
constexpr int kPfKKeys = kPfN / 2;
constexpr int kPfKChunkBytes = kPfKKeys * 128;             // [64 keys][64 dims] f16: 8192
constexpr int kPfKTileBytes = 4 * kPfKChunkBytes;          // 32768
constexpr int kPfKSlots = 3;
constexpr int kPfVDims = kHeadDim / 2;
constexpr int kPfVChunkBytes = kPfN * 128;                 // [128 keys][64 dims]: 16384
constexpr int kPfVTileBytes = 2 * kPfVChunkBytes;          // 32768
constexpr int kPfVSlots = 2;
// 224 KB of dynamic shared memory + < 3 KB static = the 227 KB an sm_100 CTA may use
constexpr int kPfSmemBytes = kPfQBytes + kPfKSlots * kPfKTileBytes + kPfVSlots * kPfVTileBytes;
constexpr int kPfBoxBytes = kPfM * 128;                    // [128 rows][32 dims] f32 of gate or output
constexpr int kPfThreads = 352;           // 8 softmax warps, K TMA, MMA, V TMA warps
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTmemO = 0;            // columns [0, 256): output accumulator
constexpr uint32_t kTmemS = 256;          // columns [256, 384): the scores of one tile
constexpr uint32_t kTmemP = 384;          // columns [384, 512): two buffers of 64 for the f16 P
constexpr float kLazyThreshold = 8.0f;    // log2 units
constexpr int kPfMaxSplits = 20;          // key splits of a tile at most
constexpr int kPfMaxParts = 256;          // parts of a balanced launch at most
constexpr int kPfMaxRecords = 7;          // of a unit there
constexpr int kPfRecAcc = 8 * 8 * kPfM;   // a CTA's record there: float4 [32 dims][4 dims][row], then (m, l) [row]
constexpr size_t kPfRecBytes = (size_t)kPfRecAcc * 16 + kPfM * 8;
// A CTA's 128 query rows: one head of 128 tokens (kHeads 1), or the three heads of half a KV head's group of 42
// tokens, token by token (kHeads 3; two rows stay empty). The pair's CTAs serve the same tokens: two heads, or all
// six of the group.
constexpr int pf_tokens(int heads) { return heads == 1 ? kPfM : kPfM / heads; }

struct PrefillArgs {
  alignas(64) CUtensorMap tm_k;
  alignas(64) CUtensorMap tm_v;
  const float *q;
  const float *gate;     // optional [n_q][n_head][256]
  const int32_t *pos;    // device, one per query token
  int n_q;
  int n_head;
  float qscale;          // scale * log2(e)
  alignas(64) CUtensorMap tm_g;  // f32 rows of the gate and the output: boxes of [tokens][heads][32 dims], 128-byte swizzle
  alignas(64) CUtensorMap tm_o;
  int n_rot;             // partial RoPE of the queries: dims [0, n_rot), pairs (d, d + n_rot / 2)
  float freq[32];        // rotation frequencies of the pairs
  int kv_wait;           // 1: the launch before this one (which waited for everything before it) stores cache
                         // rows: only the K / V loads wait for it. 0: the whole kernel waits for its predecessor
  int debug;             // timing experiments only (bit mask), 0 in production
  DeviceStatus *status;
  // Split over the keys (gridDim.z > 1): CTA (tile, head, z) walks only its share of the
  // key tiles and writes an un-normalised record (m, l, acc) per row instead of the
  // output; prefill_merge_kernel combines the records. Fills the SMs when n_q * n_head /
  // 128 CTAs would leave many idle.
  // Records: accumulators [n_q][n_head][gridDim.z][256] behind tm_o, then (m, l) here.
  float2 *rec_ml;        // [n_q][n_head][gridDim.z]
  // Balanced launch: the units (token tile, pair of CTAs along the heads), laid one behind the other, are cut into
  // as many equal runs of key tiles as pairs of CTAs fit the GPU, and every piece of a unit is a part for one pair.
  // A unit's first part writes the output; its other parts leave records for it and set their flags. The parts that
  // leave records come first in the grid, then the rest, longest first: as the first ones end, shortest first, each is
  // followed by what was cut off it. So a waiting CTA waits for CTAs that started before it, as long as the GPU starts
  // blocks in the order of their numbers. CUDA does not promise that; where it were otherwise, the wait's limit of two
  // seconds ends the launch, with zeros and a status word. A part covers [c0, c1) of the unit's key tiles counted from
  // the tokens at the end of `keys`; where pos[] says otherwise, the same fractions of what it says.
  float4 *rec;           // [record][CTA of the pair] of kPfRecBytes
  unsigned *flags;       // [record][CTA of the pair], zero before the launch
  int groups;            // units per token tile
  int keys;
  struct Part {
    unsigned short unit, c0, c1, rec, n_rec;   // rec: its record, or the first of the n_rec that it collects
  } parts[kPfMaxParts];
};
// Key tiles of a unit of token tile `tile`.
__host__ __device__ inline int pf_unit_tiles(int tile, int tokens, int n_q, int keys) {
  const int last = tile * tokens + tokens < n_q ? tile * tokens + tokens : n_q;
  return (keys - n_q + last - 1) / kPfN + 1;
}


// Barrier slots (8 bytes each).
// In the leader (CTA 0 of the pair) alone: KFull, VFull, Q, P, L -- what its issuing threads wait for, from
// both CTAs. In each CTA: KFree, VFree, S, O (tcgen05.commit arrives on both), R.
enum { kBarKFull = 0, kBarKFree = 6, kBarVFull = 12, kBarVFree = 14, kBarS = 16, kBarP = 18, kBarO = 22,
       kBarQ = 24, kBarR = 25, kBarL = 33, kBarC = 34, kBarG = 35, kBarT = 36, kBarCount = 37 };   // kBarP: [P buffer][64-key half of P];
                                                   // kBarR: [warp pair 0..3][tile parity];
                                                   // kBarL: the scores of a tile are in registers;
                                                   // kBarC: the queries are converted;
                                                   // kBarT: the (cos, sin) of the tile's rows are there;
                                                   // kBarG: the gate rows are in shared memory

// The softmax warps' waits park at the barrier at once instead of polling first: eight warps that poll take
// shared-memory cycles from the matrix unit, which reads Q, K and V there (512 tokens at 7680: 119.0 -> 117.5
// us a layer, 128 at 24000: 84.1 -> 83.0). The issuers' waits are on the critical path and go on polling.
__device__ __forceinline__ bool mbar_wait_parked(uint32_t bar, uint32_t parity, DeviceStatus *status, int site) {
  for (int i = 0; i < 12; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait(bar, parity, status, site);   // bounded
}
// A word that says "the record is written": set behind a barrier of the threads that wrote it.
__device__ __forceinline__ void flag_set(unsigned *flag) {
  __threadfence();
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(1u) : "memory");
}
__device__ __forceinline__ bool flag_wait(const unsigned *flag, DeviceStatus *status, int site) {
  const unsigned long long t0 = global_ns();
  for (uint32_t i = 1;; ++i) {
    unsigned x;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(flag) : "memory");
    if (x != 0) return true;
    if ((i & 63u) == 0 && global_ns() - t0 > kWaitNs) break;
  }
  if (status != nullptr && atomicExch(&status->timeout_flag, 1) == 0) status->where = site;
  return false;
}

template <int kHeads, bool kBalanced>
__global__ void __launch_bounds__(kPfThreads, 1) prefill_kernel(const __grid_constant__ PrefillArgs p) {
  constexpr int kTokens = pf_tokens(kHeads), kRows = kTokens * kHeads;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) unsigned long long s_bars[kBarCount];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_maxpos;
  __shared__ int s_abort;
  __shared__ int s_pos[kPfM];          // by token
  __shared__ float s_ref[2][kPfM];     // [tile parity][row]: the reference maximum that tile left

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // (uniform)
  pdl_launch_dependents();   // the merge pass of a key split may be scheduled under this kernel
  if (!p.kv_wait) pdl_wait();
  if (threadIdx.x == 0) RD_PF_TRACE(0, 47, 0);   // kernel entry
  const uint32_t rank = blockIdx.x & 1;
  int tile = (int)gridDim.y - 1 - (int)blockIdx.y;        // heaviest (latest) tiles first
  int head = blockIdx.x * kHeads;                         // the CTA's first head; the pair's are of one KV head
  int c0 = blockIdx.z, c1 = c0 + 1, n_cut = gridDim.z;    // parts [c0, c1) of n_cut of the keys
  if (kBalanced) {
    const PrefillArgs::Part &part = p.parts[blockIdx.x >> 1];
    tile = part.unit / p.groups;
    head = kHeads * (2 * (part.unit % p.groups) + (int)rank);
    c0 = part.c0;
    c1 = part.c1;
    n_cut = pf_unit_tiles(tile, kTokens, p.n_q, p.keys);
  }
  const bool leaves = kBalanced && c0 > 0;                // a record
  const int kvh = head / kGroup;
  const int tok0 = tile * kTokens;

  // carve-up of dynamic shared memory; 128B-swizzle atoms need the base 1 KB aligned
  const uint32_t base = smem_u32(smem_raw);
  if ((base & 1023u) != 0) {  // cannot happen with the declared alignment; refuse, do not corrupt
    if (threadIdx.x == 0 && p.status != nullptr && atomicExch(&p.status->timeout_flag, 1) == 0)
      p.status->where = 99;
    return;
  }
  const uint32_t sQ = base;
  const uint32_t sK = sQ + kPfQBytes;                       // slot s at + s * 32 KB
  const uint32_t sV = sK + kPfKSlots * kPfKTileBytes;       // slot s at + s * 32 KB
  uint8_t *gQ = smem_raw;                                   // generic pointer to sQ
  const uint32_t bars = smem_u32(s_bars), lead = cluster_addr(bars, 0);   // this CTA's barriers, the leader's

  // Requested first, so that their latency runs under the set-up below: the positions of this tile's
  // rows and, to L2, the warp's 16 query rows. (Loaded to registers here they are spilled, and the spill
  // waits for them.)
  int my_pos = -1;
  const int toks_cta = min(p.n_q - tok0, kTokens), rows_cta = toks_cta * kHeads;   // of the tile, how many exist
  const int toks_cs = toks_cta > 64 ? 128 : toks_cta > 32 ? 64 : 32;   // and how many the (cos, sin) table is made for
  float4 xa[8], xb[8];   // dims 4 lane .. + 3 and 128 + 4 lane .. + 3 of a row
  const int rows_w = rows_cta - warp * 16;   // of the warp's rows, how many exist
  auto q_at = [&](int rr) {                  // its rr-th one
    const int row = warp * 16 + rr;
    return p.q + ((size_t)(tok0 + row / kHeads) * p.n_head + head + row % kHeads) * kHeadDim;
  };
  auto load_rows = [&](int first) {
#pragma unroll
    for (int rr = 0; rr < 8; ++rr) {
      xa[rr] = xb[rr] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (first + rr < rows_w) {
        const float4 *src = reinterpret_cast<const float4 *>(q_at(first + rr));
        xa[rr] = src[lane];
        xb[rr] = src[lane + 32];
      }
    }
  };
  if (threadIdx.x < 2 * kPfM) {
    const int r = threadIdx.x & (kPfM - 1);
    if (r < rows_cta) my_pos = p.pos[tok0 + r / kHeads];
#pragma unroll
    for (int e = 0; e < 4; ++e) {   // 16 rows x 8 lines of 128 bytes
      const int rr = (lane >> 3) + 4 * e;
      if (rr < rows_w) asm volatile("prefetch.global.L2 [%0];" ::"l"(q_at(rr) + 32 * (lane & 7)));
    }
  }

  if (threadIdx.x == 0) {
    s_maxpos = -1;
    s_abort = 0;
    // Softmax warps, of both CTAs, that have a row at all: the others take no part in the loop. (Handing the
    // buffers on instead, they poll barriers in the shared memory that the matrix unit reads its operands from:
    // 24 queries at 24000 86 us a layer.)
    const int live_warps = 2 * min((rows_cta + 31) / 32, 4);
    for (int i = 0; i < kPfKSlots; ++i) {
      mbar_init(bars + 8 * (kBarKFull + i), 1);
      mbar_init(bars + 8 * (kBarKFree + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bars + 8 * (kBarVFull + i), 1);
      mbar_init(bars + 8 * (kBarVFree + i), 1);
      mbar_init(bars + 8 * (kBarS + i), 1);
      mbar_init(bars + 8 * (kBarP + 2 * i), live_warps);       // one elected lane per softmax warp of the
      mbar_init(bars + 8 * (kBarP + 2 * i + 1), live_warps);   // tile's set (both CTAs), per 64-key half of P
      mbar_init(bars + 8 * (kBarO + i), 1);
    }
    for (int i = 0; i < 8; ++i) mbar_init(bars + 8 * (kBarR + i), 1);
    mbar_init(bars + 8 * kBarL, live_warps);
    mbar_init(bars + 8 * kBarQ, 16);   // one per converting warp (both CTAs)
    mbar_init(bars + 8 * kBarT, 9);    // the CTA's warps, and the bytes of the peer's half
    mbar_init(bars + 8 * kBarC, 8);
    mbar_init(bars + 8 * kBarG, 1);
    fence_barrier_init();
    mbar_expect_tx(bars + 8 * kBarT, p.n_rot == 64 ? toks_cs / 2 * 32 * 8 : 0);
  }
  if (warp == 9) {  // TMEM: 512 columns for this CTA (one CTA per SM: no contention)
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) RD_PF_TRACE(0, 47, 1);   // barriers + TMEM allocated
  if (warp < 8) load_rows(0);

  // ---- the last key any row of this tile attends ----
  if (threadIdx.x < kPfM) {
    int mx = my_pos;
    if (kHeads == 1 || threadIdx.x % kHeads == 0) s_pos[threadIdx.x / kHeads] = my_pos;
    if (kHeads > 1 && threadIdx.x > kTokens) s_pos[threadIdx.x] = -1;   // (the table is made for more tokens)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) atomicMax(&s_maxpos, mx);
  }
  tc_fence_before();
  cluster_sync();   // the pair's barriers are initialised, its tensor memory allocated
  if (threadIdx.x == 0) RD_PF_TRACE(0, 47, 2);   // positions known
  tc_fence_after();
  const uint32_t tmem = s_tmem_base;
  const int maxpos = s_maxpos;
  const int nt_all = maxpos >= 0 ? maxpos / kPfN + 1 : 0;  // key tiles the rows of this tile attend
  const int jt0 = (int)(((int64_t)nt_all * c0) / n_cut);        // this CTA's share of them
  const int nt = (int)(((int64_t)nt_all * c1) / n_cut) - jt0;

  // ---- prologue: the Q tile as f16 in the swizzled K-major layout ----
  // f32 rows -> partial RoPE -> x scale * log2(e) -> f16 in the swizzled layout, warps 0-7. (A pre-pass
  // that wrote rotated f16 queries for all heads cost its own 6 us and a second trip to memory: 15400
  // cycles from entry to the first S; the f32 rows by bulk copies or a tensor-map box: 13300; here 11000, of
  // which the loads of 128 KB take 2600 to issue.)
  if (warp < 8) {
    // thread (row r, h) rotates dims 0..63 of its row; they pass through V slot 1 as f32, 16-byte chunk q of
    // a row at q ^ (r & 15)
    float *stage = reinterpret_cast<float *>(gQ + (sV - sQ) + kPfVTileBytes);
    const int r = threadIdx.x & (kPfM - 1), h = threadIdx.x >> 7;
    const uint32_t qrow = sQ + r * 128, swz = (uint32_t)(r & 7) << 4;   // (sub-tile 0: dims 0..63)
    // four dims of a row: sub-tile q4 / 16, 16-byte chunk q4 / 2, half q4 & 1
    auto put4 = [&](int rr, int q4, const float4 &x) {
      sts64(sQ + (q4 >> 4) * (kPfM * 128) + rr * 128 + (((uint32_t)((q4 >> 1) & 7) ^ (rr & 7)) << 4) + (q4 & 1) * 8,
            pack_h2(x.x * p.qscale, x.y * p.qscale), pack_h2(x.z * p.qscale, x.w * p.qscale));
    };
    auto convert = [&](int first) {
      if (rows_cta <= 32 * (warp >> 1)) return;   // (no row of a whole softmax warp exists: nobody reads the scores)
#pragma unroll
      for (int k = 0; k < 8; ++k) put4(warp * 16 + first + k, lane + 32, xb[k]);
      if (p.n_rot > 0 && lane < 16) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int rr = warp * 16 + first + k;
          *reinterpret_cast<float4 *>(stage + rr * 64 + ((lane ^ (rr & 15)) << 2)) = xa[k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) put4(warp * 16 + first + k, lane, xa[k]);
      }
    };
    if (threadIdx.x == 0) RD_PF_TRACE(0, 46, 2);
    convert(0);
    if (threadIdx.x == 0) RD_PF_TRACE(0, 46, 3);
    load_rows(8);
    if (threadIdx.x == 0) RD_PF_TRACE(0, 46, 4);
    // (cos, sin) of all rows and pairs, while those are on their way: the two CTAs of the pair serve the same
    // tokens, each computes half for both (16 sincosf per thread took 4200 cycles). [pair][token] in V slot 0.
    const uint32_t cs0 = sV;
    const float *cs = reinterpret_cast<const float *>(gQ + (sV - sQ));
    if (p.n_rot == 64) {
      const int id = (int)rank * 256 + threadIdx.x, tr = id & (toks_cs - 1);   // token, and toks_cs / 16 pairs of it
      const int tp = id / toks_cs * (toks_cs / 16);
      const float fpos = (float)s_pos[tr];
      const uint32_t peer = cluster_addr(cs0, rank ^ 1), peer_bar = cluster_addr(bars + 8 * kBarT, rank ^ 1);
#pragma unroll 1
      for (int i = 0; i < toks_cs / 16; i += 2) {
        float2 v[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) sincosf(fpos * p.freq[tp + i + e], &v[e].y, &v[e].x);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t at = 8u * ((tp + i + e) * kPfM + tr);
          sts64(cs0 + at, __float_as_uint(v[e].x), __float_as_uint(v[e].y));
          // (completes on the peer's barrier by bytes: no fence, no remote arrive)
          asm volatile(
              "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(peer + at),
              "r"(__float_as_uint(v[e].x)), "r"(__float_as_uint(v[e].y)), "r"(peer_bar)
              : "memory");
        }
      }
      __syncwarp();
      if (threadIdx.x == 0) RD_PF_TRACE(0, 46, 5);
      if (lane == 0) mbar_arrive(bars + 8 * kBarT);
    }
    convert(8);
    if (threadIdx.x == 0) RD_PF_TRACE(0, 46, 0);
    if (threadIdx.x == 0) RD_PF_TRACE(0, 46, 1);
    if (p.n_rot > 0) {
      if (p.n_rot == 64 && !mbar_wait(bars + 8 * kBarT, 0, p.status, 24)) s_abort = 1;
      asm volatile("bar.sync 2, 256;" ::: "memory");
      auto chunk = [&](int q) { return *reinterpret_cast<const float4 *>(stage + r * 64 + ((q ^ (r & 15)) << 2)); };
      if (p.n_rot == 64) {
        float4 ca[4], cb[4];
        float2 cc[16];
#pragma unroll
        for (int k = 0; k < 4; ++k) ca[k] = chunk(4 * h + k), cb[k] = chunk(8 + 4 * h + k);
#pragma unroll
        for (int e = 0; e < 16; ++e) cc[e] = reinterpret_cast<const float2 *>(cs)[(16 * h + e) * kPfM + r / kHeads];
#pragma unroll
        for (int k = 0; k < 4; ++k) {   // four pairs
          const float4 a = ca[k], b = cb[k];
          const float x0[4] = {a.x, a.y, a.z, a.w}, x1[4] = {b.x, b.y, b.z, b.w};
          float y0[4], y1[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 c = cc[4 * k + e];
            y0[e] = __fsub_rn(__fmul_rn(x0[e], c.x), __fmul_rn(x1[e], c.y)) * p.qscale;
            y1[e] = __fadd_rn(__fmul_rn(x0[e], c.y), __fmul_rn(x1[e], c.x)) * p.qscale;
          }
          const uint32_t lo = (uint32_t)(2 * h + (k >> 1)) << 4, hi = lo + 64, half = (k & 1) * 8;
          sts64(qrow + (lo ^ swz) + half, pack_h2(y0[0], y0[1]), pack_h2(y0[2], y0[3]));
          sts64(qrow + (hi ^ swz) + half, pack_h2(y1[0], y1[1]), pack_h2(y1[2], y1[3]));
        }
      } else {   // other rotary sizes: value by value
        auto get = [&](int d) { return stage[r * 64 + (((d >> 2) ^ (r & 15)) << 2) + (d & 3)]; };
        auto put = [&](int d, float x) {
          const unsigned short hx = __half_as_ushort(__float2half_rn(x * p.qscale));
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(qrow + (((uint32_t)(d >> 3) << 4) ^ swz) + 2 * (d & 7)), "h"(hx)
                       : "memory");
        };
        const int nh = p.n_rot / 2;
#pragma unroll 1
        for (int d = h; d < nh; d += 2) {
          float c, sn;
          sincosf((float)my_pos * p.freq[d], &sn, &c);
          const float x0 = get(d), x1 = get(d + nh);
          put(d, __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, sn)));
          put(d + nh, __fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, c)));
        }
#pragma unroll 1
        for (int d = p.n_rot + h; d < 64; d += 2) put(d, get(d));
      }
    }
    fence_proxy_async();  // generic-proxy accesses before those of the tensor core and the copies
    __syncwarp();
    if (lane == 0) {
      mbar_arrive_peer(lead + 8 * kBarQ);   // the S MMAs wait for all 16 warps
      mbar_arrive(bars + 8 * kBarC);
    }
    if (threadIdx.x == 0) RD_PF_TRACE(0, 47, 3);   // this warp's Q rows converted
  }

  const bool with_gate = p.gate != nullptr && gridDim.z == 1 && !leaves;
  float l_run = 0.f;                 // softmax threads: row sum
  float m_ref = -1.0e30f;            //                  reference maximum (log2 units)

  if (warp >= 8) {
  if (warp == 8) {
    // =============================== K producer ====================================
    // this CTA's half of tile j (64 keys) into slot j % 3; both CTAs' copies complete on the leader's barrier
    if (lane == 0) {
      if (p.kv_wait) pdl_wait();   // the pre-pass of this call appended rows to the caches
      int slot = 0, use = 0;
      for (int j = 0; j < nt; ++j) {
        if (use > 0 && !mbar_wait(bars + 8 * (kBarKFree + slot), (use - 1) & 1, p.status, 11)) {
          s_abort = 1;
          break;
        }
        if (*(volatile int *)&s_abort) break;
        if (rank == 0) mbar_expect_tx(bars + 8 * (kBarKFull + slot), 2 * kPfKTileBytes);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          tma_load_2d_pair(sK + slot * kPfKTileBytes + c * kPfKChunkBytes, &p.tm_k, kvh * kHeadDim + 64 * c,
                           (jt0 + j) * kPfN + (int)rank * kPfKKeys, lead + 8 * (kBarKFull + slot));
        if (++slot == kPfKSlots) {
          slot = 0;
          ++use;
        }
      }
    }
    if (with_gate) {
      // Q and the K ring are free once the last S has been computed: the gate rows come into them (128
      // KB) under the last tile's softmax and P V. (Loaded to registers between the epilogue's
      // stores, a few at a time, their latency was most of it: 15000 of 18000 cycles.)
      // (lane 0 has waited for every earlier use of that K slot: a parity two uses old cannot pass)
      if (lane == 0) {
        const bool ok =
            mbar_wait(bars + 8 * kBarC, 0, p.status, 26) &&
            (nt == 0 ||
             mbar_wait(bars + 8 * (kBarKFree + (nt - 1) % kPfKSlots), ((nt - 1) / kPfKSlots) & 1, p.status, 27));
        if (ok) {
          mbar_expect_tx(bars + 8 * kBarG, kRows * kHeadDim * 4);
          for (int c = 0; c < 8; ++c)
            tma_load_3d(sQ + c * kPfBoxBytes, &p.tm_g, 32 * c, head, tok0, bars + 8 * kBarG);
        } else {
          s_abort = 1;
          mbar_arrive(bars + 8 * kBarG);   // nobody waits for long
        }
      }
    }
  } else if (warp == 10) {
    // =============================== V producer ====================================
    // this CTA's half of tile j (128 of the 256 dims) into slot j % 2
    if (with_gate && lane == 1) {
      // the gate rows that the epilogue multiplies with, on their way to L2 once the queries have arrived
      // (before, the two would share the memory's bandwidth and the queries come first)
      mbar_wait(bars + 8 * kBarC, 0, nullptr, 0);
      for (int c = 0; c < 8; ++c) tma_prefetch_3d(&p.tm_g, 32 * c, head, tok0);
    }
    if (lane == 0) {
      if (p.kv_wait) pdl_wait();
      for (int j = 0; j < nt; ++j) {
        const int slot = j & 1;
        if (j == 0 ? !mbar_wait(bars + 8 * kBarC, 0, p.status, 23)   // the query conversion has left the slots
                   : j >= 2 && !mbar_wait(bars + 8 * (kBarVFree + slot), ((j >> 1) - 1) & 1, p.status, 22)) {
          s_abort = 1;
          break;
        }
        if (*(volatile int *)&s_abort) break;
        if (rank == 0) mbar_expect_tx(bars + 8 * (kBarVFull + slot), 2 * kPfVTileBytes);
#pragma unroll
        for (int c = 0; c < 2; ++c)
          tma_load_2d_pair(sV + slot * kPfVTileBytes + c * kPfVChunkBytes, &p.tm_v,
                           kvh * kHeadDim + (int)rank * kPfVDims + 64 * c, (jt0 + j) * kPfN, lead + 8 * (kBarVFull + slot));
      }
    }
  } else if (warp == 9) {
    // ============ MMA issuer: S = Q K^T of tile i, then O += P V of tile i - 2 ============
    // One warp, one order: the tensor core works its queue off in order, so a tile's scores are ready after
    // 1024 cycles and the softmax warps copy them to registers under the P V behind them. The warp stays
    // converged and elect.sync picks the lane (see elect_one): issued by "lane 0" an instruction took 70 to
    // 110 cycles of moves to uniform registers, as long as the tensor core runs it. Then each contraction
    // needed a thread of its own, their instructions lay alternately in the queue, scores came 2300 to 2800 cycles
    // after the request and the queue ran dry while they were copied: 2950 cycles a tile with all SMs at work,
    // now 2060 (512 tokens at 7680: 1880 -> 1775 us for 16 layers, at the power cap; 8192 at 0: 825 -> 767).
    if (rank == 0) {
      constexpr uint32_t idesc_s = idesc_f16(2 * kPfM, kPfN, false);
      constexpr uint32_t idesc_o = idesc_f16(2 * kPfM, kHeadDim, true);
      // Descriptors differ only in the 16-byte-granular start address (low 14 bits, and
      // every address here is below 256 KB), so each one is a base plus a constant.
      const uint64_t dq = smem_desc(sQ, 16, 1024);
      const uint64_t dk = smem_desc(sK, 16, 1024);
      const uint64_t dv = smem_desc(sV, kPfVChunkBytes, 1024);
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      const int n = __shfl_sync(0xffffffffu, nt, 0);
      auto wait = [&](int bar, int parity, int site) {
        return __all_sync(0xffffffffu, mbar_wait(bars + 8 * bar, parity, p.status, site));
      };
      bool ok = wait(kBarQ, 0, 18);  // both Q tiles are there
      tc_fence_after();
      int slot = 0, use = 0;
      for (int i = 0; i < n + 2 && ok; ++i) {
        if (i < n) {
          RD_PF_TRACE(2, i, 0);
          if (!wait(kBarKFull + slot, use & 1, 12)) {
            ok = false;
            break;
          }
          RD_PF_TRACE(2, i, 1);
          // the softmax warps of tile i - 1 (both CTAs) have its scores in registers
          if (i >= 1 && !wait(kBarL, (i - 1) & 1, 15)) {
            ok = false;
            break;
          }
          tc_fence_after();
          RD_PF_TRACE(2, i, 3);
          // per 64-dim chunk c: A = Q sub-tile c ([128 rows][64 dims] in each CTA), B = K chunk c ([64
          // keys][64 dims] in each), K-major with 8-row groups 1 KB apart; four steps of 16 dims
          if (elect_one()) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const uint64_t a0 = dq + (uint64_t)((c * (kPfM * 128)) >> 4);
              const uint64_t b0 = dk + (uint64_t)((slot * kPfKTileBytes + c * kPfKChunkBytes) >> 4);
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                tc_mma2_f16(tm + kTmemS, a0 + (uint64_t)(2 * kk), b0 + (uint64_t)(2 * kk), idesc_s,
                            (c > 0 || kk > 0) ? 1u : 0u);
            }
            tc_commit2(bars + 8 * (kBarS + (i & 1)));
            tc_commit2(bars + 8 * (kBarKFree + slot));  // the tile can be refilled
          }
          __syncwarp();
          RD_PF_TRACE(2, i, 4);
          if (++slot == kPfKSlots) {
            slot = 0;
            ++use;
          }
          RD_PF_TRACE(2, i, 2);
        }
        if (i < 2) continue;
        const int j = i - 2, st = j & 1;
        RD_PF_TRACE(3, j, 0);
        if (!wait(kBarVFull + st, (j >> 1) & 1, 19)) {
          ok = false;
          break;
        }
        for (int u = 0; u < 2 && ok; ++u) {
          // P arrives in two halves of 64 keys: P V of the first runs while the softmax
          // threads are still on the second
          if (!wait(kBarP + 2 * st + u, (j >> 1) & 1, 13)) {
            ok = false;
            break;
          }
          RD_PF_TRACE(3, j, 1 + 2 * u);
          tc_fence_after();
          // A = P(j) from TMEM (16 keys = 8 columns per step), B = V MN-major, 128 of the 256 dims in each
          // CTA: 64-dim groups 16 KB apart (LBO), 8-key groups 1 KB apart (SBO); 4 steps of 16 keys
          const uint64_t dvs = dv + (uint64_t)((st * kPfVTileBytes + u * 8192) >> 4);
          const uint32_t a_p = tm + kTmemP + 64 * st + 32 * u;
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              tc_mma2_f16_ts(tm + kTmemO, a_p + 8 * kk, dvs + (uint64_t)((kk * 2048) >> 4), idesc_o,
                             (j > 0 || u > 0 || kk > 0) ? 1u : 0u);
            if (u == 1) {
              tc_commit2(bars + 8 * (kBarVFree + st));  // the V tile can be refilled
              tc_commit2(bars + 8 * (kBarO + st));      // P buffer reusable, O settled
            }
          }
          __syncwarp();
        }
        if (!ok) break;
        RD_PF_TRACE(3, j, 2);
      }
      if (!ok) s_abort = 1;
    }
  }
  } else {
    // ========= softmax: thread = (row r, tile parity): warps 0-3 take the even key =========
    // tiles of this CTA, warps 4-7 the odd ones, a whole 128-key row of scores per thread.
    // The two sets run one tile apart, so the tensor-memory loads, the maxima and the waits
    // of tile j + 1 overlap the exponentials of tile j. What the tiles of a row share is the
    // reference maximum of the one accumulator: it is handed from tile to tile through
    // s_ref and one mbarrier per (warp pair, parity) -- after a tile's maxima are known,
    // before its exponentials.
    const int r = threadIdx.x & (kPfM - 1), set = threadIdx.x >> 7;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t bar_ref = bars + 8 * (kBarR + 2 * (warp & 3));
    bool ok = true;
    const bool live = 32 * (warp & 3) < rows_cta;   // (the barriers count the warps that have a row)
    // Rows past the last query see every key: nobody reads what they give, and a mask on their account would
    // be a mask on every tile (24 queries at 16000: 94 us a layer with it).
    const int last_key = r < rows_cta ? my_pos : 0x7fffffff;
    for (int j = set; live && j < nt && ok; j += 2) {
      const int st = set;   // tile j's P buffer: j & 1
      if ((threadIdx.x & 127) == 0) RD_PF_TRACE(set, j, 0);
      // the reference tile j - 1 left: its set published it right after its own maxima,
      // long before this tile's scores are ready -- fetched first, off the critical path
      float m_prev = -1.0e30f;
      if (j > 0) {
        if (!mbar_wait_parked(bar_ref + 8 * ((j - 1) & 1), ((j - 1) >> 1) & 1, p.status, 20)) { ok = false; break; }
        m_prev = s_ref[(j - 1) & 1][r];
      }
      if (!mbar_wait_parked(bars + 8 * (kBarS + st), (j >> 1) & 1, p.status, 14)) { ok = false; break; }
      tc_fence_after();
      if ((threadIdx.x & 127) == 0) RD_PF_TRACE(set, j, 1);
      uint32_t sc[4][32];
      const uint32_t scol = lane_addr + kTmemS, pcol = lane_addr + kTmemP + 64 * st;
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(scol + 32 * c, sc[c]);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_peer(lead + 8 * kBarL);   // S of tile j + 1 can be computed
      if ((threadIdx.x & 127) == 0) RD_PF_TRACE(set, j, 2);
      const int key0 = (jt0 + j) * kPfN;
      // only tiles that reach past some row's last key need the causal mask
      if (__any_sync(0xffffffffu, key0 + kPfN - 1 > last_key)) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + 32 * c + i > last_key) sc[c][i] = 0xff800000u;  // -inf
      }
      // eight independent chains of three-input maxima
      float mx[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) mx[k] = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          mx[(i >> 1) & 7] = max3(mx[(i >> 1) & 7], __uint_as_float(sc[c][i]), __uint_as_float(sc[c][i + 1]));
      const float mt = fmaxf(max3(mx[0], mx[1], mx[2]), fmaxf(max3(mx[3], mx[4], mx[5]), fmaxf(mx[6], mx[7])));
      const bool grow = __any_sync(0xffffffffu, mt > m_prev + kLazyThreshold);
      const float m_new = grow ? fmaxf(m_prev, mt) : m_prev;
      s_ref[j & 1][r] = m_new;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ref + 8 * (j & 1));
      if ((threadIdx.x & 127) == 0) RD_PF_TRACE(set, j, 3);
      l_run *= ex2(m_ref - m_new);   // this set's sum moves to the new reference (m_ref: its last one)
      m_ref = m_new;
      if (grow && j > 0) {
        // O is rescaled in tensor memory: P V of tile j - 1 must be done, and no later one
        // can start before this tile's P arrives
        const float f = ex2(m_prev - m_new);   // 1 for rows that keep their reference
        if (!mbar_wait_parked(bars + 8 * (kBarO + ((j - 1) & 1)), ((j - 1) >> 1) & 1, p.status, 17)) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < kHeadDim / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(lane_addr + kTmemO + 32 * c, o);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
          tmem_st32(lane_addr + kTmemO + 32 * c, o);
        }
        tmem_wait_st();
      }
      // P = 2^(s - m_ref) as f16 pairs: key k of row r becomes half k & 1 of column k / 2 (the A
      // operand of P V, read from TMEM)
      // (s - m) and the row sum go through the packed f32x2 adds, two scores per
      // instruction: measured alone, one warp then needs ~1200 cycles per 128-score row
      // (the 128 exponentials alone are 1024 on the special-function unit) against ~1600
      // with scalar adds
      // (P V of tile j - 2 has read this buffer)
      if (j >= 2 && !mbar_wait_parked(bars + 8 * (kBarO + st), ((j - 2) >> 1) & 1, p.status, 21)) { ok = false; break; }
      tc_fence_after();
      unsigned long long neg_m = f2_pack(-m_new, -m_new);
      unsigned long long ls2[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pw[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float x0, x1;
          f2_unpack(f2_add(f2_pack(__uint_as_float(sc[c][2 * i]), __uint_as_float(sc[c][2 * i + 1])), neg_m), x0, x1);
          if (!(RD_PF_DEBUG(p) & 1)) {
            x0 = ex2(x0);
            x1 = ex2(x1);
          }
          ls2[i & 3] = f2_add(ls2[i & 3], f2_pack(x0, x1));
          pw[i] = (RD_PF_DEBUG(p) & 2) ? __float_as_uint(x0) : pack_h2(x0, x1);
        }
        if (!(RD_PF_DEBUG(p) & 16)) tmem_st16(pcol + 16 * c, pw);
        else if (pw[0] == 0x12345678u && pw[7] == 0x9abcdefu) l_run += 1.f;   // keeps the values live
        if (c == 1) {   // the first 64 keys of P are complete: hand them to the P V issuer
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_peer(lead + 8 * (kBarP + 2 * st));
          // keeps the second half's arithmetic behind the hand-over (the compiler would
          // otherwise hoist all 128 exponentials above the first store)
          asm volatile("mov.b64 %0, %0;" : "+l"(neg_m)::"memory");
        }
      }
      {
        float a0, a1, a2, a3;
        f2_unpack(f2_add(ls2[0], ls2[1]), a0, a1);
        f2_unpack(f2_add(ls2[2], ls2[3]), a2, a3);
        l_run += (a0 + a1) + (a2 + a3);
      }
      if ((threadIdx.x & 127) == 0) RD_PF_TRACE(set, j, 4);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_peer(lead + 8 * (kBarP + 2 * st + 1));
      if ((threadIdx.x & 127) == 0) RD_PF_TRACE(set, j, 5);
    }
    if (live && ok && nt > 0 && !mbar_wait_parked(bars + 8 * (kBarO + ((nt - 1) & 1)), ((nt - 1) >> 1) & 1, p.status, 16))
      ok = false;
    if (!ok) s_abort = 1;
    tc_fence_after();
  }

  cluster_sync();   // both CTAs are done with each other's barriers, shared and tensor memory
  const bool aborted = s_abort != 0;
  // the two sets' row sums, each with the reference it is expressed in: [set][sum,
  // reference][row], over the third K slot (the gate rows lie in Q and the first two)
  float (*s_fin)[2][kPfM] = reinterpret_cast<float (*)[2][kPfM]>(smem_raw + kPfQBytes + 2 * kPfKTileBytes);
  if (warp < 8) {
    s_fin[threadIdx.x >> 7][0][threadIdx.x & (kPfM - 1)] = l_run;
    s_fin[threadIdx.x >> 7][1][threadIdx.x & (kPfM - 1)] = m_ref;
  }
  __syncthreads();
  if (threadIdx.x == 0) RD_PF_TRACE(0, 47, 4);   // main loop done, sums exchanged

  // ---- epilogue ----
  if (warp < 8) {
    // warpgroup ch stores output columns [64*(2c+ch), +64), c = 0..1, through its own
    // staging tile and named barrier
    const int r = threadIdx.x & (kPfM - 1), ch = threadIdx.x >> 7, gt = threadIdx.x & (kPfM - 1);
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    // both sums at the reference the last tile left (a set without tiles: sum 0)
    const float m_fin = nt > 0 ? s_ref[(nt - 1) & 1][r] : -1.0e30f;
    const float l_tot = s_fin[0][0][r] * ex2(s_fin[0][1][r] - m_fin) + s_fin[1][0][r] * ex2(s_fin[1][1][r] - m_fin);
    const bool rec_mode = gridDim.z > 1;   // un-normalised records for prefill_merge_kernel
    const bool have = nt > 0 && !aborted;
    // Where a unit's parts are added up, a row without a key in this one gives nothing: its accumulators may be
    // 0 x infinity, from values behind the row's last key.
    const bool empty = !have || (kBalanced && l_tot == 0.f);
    float l_sum = l_tot;   // of the unit's parts
    // Weights of the parts: this one's, then [part][row] in the third K slot, behind the row sums.
    float w_own = 1.f;
    bool lost = false;
    float (*s_w)[kPfM] = reinterpret_cast<float (*)[kPfM]>(smem_raw + kPfQBytes + 2 * kPfKTileBytes + 2048) + ch * kPfMaxRecords;
    int n_other = 0;
    const float4 *others = nullptr;   // records, 2 apart
    if (kBalanced && !leaves) {
      const PrefillArgs::Part &part = p.parts[blockIdx.x >> 1];
      n_other = part.n_rec;
      others = p.rec + (2 * (size_t)part.rec + rank) * (kPfRecBytes / 16) + r;
    }
    if (n_other > 0) {
      pdl_wait();   // (the flags are zeroed by the launch before this one; its end was waited for long ago)
      const bool there = lane >= n_other || flag_wait(p.flags + 2 * (p.parts[blockIdx.x >> 1].rec + lane) + rank, p.status, 29);
      lost = !__all_sync(0xffffffffu, there);
      __syncwarp();   // what one lane's acquire has seen is seen by the others from here on (a vote orders no memory)
      float m_all = m_fin;
      for (int i = 0; i < n_other; ++i)
        m_all = fmaxf(m_all, __ldcg(reinterpret_cast<const float2 *>(others - r + 2 * i * (kPfRecBytes / 16) + kPfRecAcc) + r).x);
      w_own = ex2(m_fin - m_all);
      l_sum *= w_own;
      for (int i = 0; i < n_other; ++i) {
        const float2 ml = __ldcg(reinterpret_cast<const float2 *>(others - r + 2 * i * (kPfRecBytes / 16) + kPfRecAcc) + r);
        const float w = ex2(ml.x - m_all);
        s_w[i][r] = w;   // (read by this thread only)
        l_sum = fmaf(ml.y, w, l_sum);
      }
    }
    const float inv = (l_sum > 0.f && !aborted && !lost) ? (rec_mode ? 1.0f : 1.0f / l_sum) : 0.f;
    // column of the first value in a head's output, or in the accumulators of its records
    const int col0 = rec_mode ? (int)blockIdx.z * kHeadDim : 0;
    if (rec_mode && ch == 0 && r < rows_cta) {
      // (m, l) of this row's record, in natural-log units
      const bool some = have && l_tot > 0.f;
      p.rec_ml[((size_t)(tok0 + r / kHeads) * p.n_head + head + r % kHeads) * gridDim.z + blockIdx.z] =
          some ? make_float2(m_fin * 0.6931471805599453f, l_tot) : make_float2(-INFINITY, 0.f);
    }
    if (leaves) {   // 512 contiguous bytes per store of a warp
      const int slot = p.parts[blockIdx.x >> 1].rec;
      float4 *rec = p.rec + (2 * (size_t)slot + rank) * (kPfRecBytes / 16) + r;
      if (ch == 0) reinterpret_cast<float2 *>(rec - r + kPfRecAcc)[r] = have ? make_float2(m_fin, l_tot) : make_float2(-1.0e30f, 0.f);
#pragma unroll 1
      for (int b = ch; b < 8 && 32 * (warp & 3) < rows_cta; b += 2) {
        uint32_t o[32];
        if (have) {
          tmem_ld32(lane_addr + kTmemO + 32 * b, o);
          tmem_wait_ld();
        }
        if (empty) {
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = 0u;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
          __stcg(rec + (b * 8 + q) * kPfM, make_float4(__uint_as_float(o[4 * q]), __uint_as_float(o[4 * q + 1]),
                                                       __uint_as_float(o[4 * q + 2]), __uint_as_float(o[4 * q + 3])));
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
      if (threadIdx.x == 0) flag_set(p.flags + 2 * slot + rank);
    } else {
      // O / l (x sigmoid(gate)) in place over the gate rows, 32 columns (a box of 128-byte swizzled rows)
      // at a time, each box stored by TMA while the next is computed. What bounds it: the 32 bytes a
      // cycle that an SM writes (4096 cycles) and 1.5 special functions per gate value (3072).
      float4 x[8];   // 32 values of a record
      auto fetch = [&](int b, int i) {
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] = __ldcg(others + 2 * i * (kPfRecBytes / 16) + (b * 8 + q) * kPfM);
      };
      if (kBalanced && n_other > 0) fetch(ch, 0);
      if (with_gate) mbar_wait(bars + 8 * kBarG, 0, p.status, 28);
#pragma unroll 1
      for (int b = ch; b < 8; b += 2) {
        uint32_t o[32];
        if (32 * (warp & 3) >= rows_cta) {   // none of the warp's rows exists: only the barrier below
          asm volatile("bar.sync %0, 128;" ::"r"(3 + ch) : "memory");
          continue;
        }
        if (have) {
          tmem_ld32(lane_addr + kTmemO + 32 * b, o);
          tmem_wait_ld();
        }
        if (empty) {
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = 0u;
        }
        if (kBalanced && n_other > 0) {
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * w_own);
#pragma unroll 1
          for (int i = 0; i < n_other; ++i) {
            const float w = s_w[i][r];
            float4 y[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) y[q] = x[q];
            // the next values are on their way while these, or the rest of the box, are worked on
            if (i + 1 < n_other) fetch(b, i + 1);
            else if (b + 2 < 8) fetch(b + 2, 0);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              o[4 * q] = __float_as_uint(fmaf(y[q].x, w, __uint_as_float(o[4 * q])));
              o[4 * q + 1] = __float_as_uint(fmaf(y[q].y, w, __uint_as_float(o[4 * q + 1])));
              o[4 * q + 2] = __float_as_uint(fmaf(y[q].z, w, __uint_as_float(o[4 * q + 2])));
              o[4 * q + 3] = __float_as_uint(fmaf(y[q].w, w, __uint_as_float(o[4 * q + 3])));
            }
          }
        }
        const uint32_t brow = sQ + b * kPfBoxBytes + r * 128;
        uint32_t nan = 0;   // columns of the row with a NaN gate
        auto box_at = [&](int e) { return ((uint32_t)((e >> 2) ^ (r & 7)) << 4) + 4 * (e & 3); };
        if (with_gate) {
          float g[32];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint4 x = lds128(brow + ((uint32_t)(q ^ (r & 7)) << 4));
            g[4 * q] = __uint_as_float(x.x);
            g[4 * q + 1] = __uint_as_float(x.y);
            g[4 * q + 2] = __uint_as_float(x.z);
            g[4 * q + 3] = __uint_as_float(x.w);
          }
          // A NaN gate makes its output NaN, as in the merge of a key split. (The cap on e^-g below takes a NaN, and
          // the pair's other value must not see it. Rolled loops: a kernel that runs once pays for every line of
          // instructions it fetches; with these 32 values unrolled 512 tokens at 0 took 0.37 us a layer longer.)
          unsigned long long sum[2] = {0ull, 0ull};   // NaN if one of the gates is
#pragma unroll
          for (int e = 0; e < 16; ++e) sum[e & 1] = f2_add(sum[e & 1], f2_pack(g[2 * e], g[2 * e + 1]));
          float n0, n1;
          f2_unpack(f2_add(sum[0], sum[1]), n0, n1);
          if (n0 + n1 != n0 + n1) {
#pragma unroll 1
            for (int e = 0; e < 32; ++e)
              nan |= (uint32_t)((lds32(brow + box_at(e)) & 0x7fffffffu) > 0x7f800000u) << e;
          }
          // Branch-free from here to the stores: 32 independent chains.
          // One reciprocal for two values; e^-g is capped at 2^60. Approximate exp and reciprocal: ~1e-6 relative
#pragma unroll
          for (int e = 0; e < 32; ++e) g[e] = 1.0f + ex2(fminf(g[e] * -1.4426950408889634f, 60.f));
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float rr = rcp_approx(g[e] * g[e + 1]) * inv;
            o[e] = __float_as_uint(__uint_as_float(o[e]) * (g[e + 1] * rr));
            o[e + 1] = __float_as_uint(__uint_as_float(o[e + 1]) * (g[e] * rr));
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * inv);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
          sts128(brow + ((uint32_t)(q ^ (r & 7)) << 4), o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
#pragma unroll 1
        for (; nan != 0; nan &= nan - 1)
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(brow + box_at(__ffs(nan) - 1)), "r"(0x7fffffffu) : "memory");
        fence_proxy_async();
        asm volatile("bar.sync %0, 128;" ::"r"(3 + ch) : "memory");
        if (gt == 0) {
          tma_store_3d(&p.tm_o, sQ + b * kPfBoxBytes, col0 + 32 * b, head, tok0);   // tokens past n_q are clipped
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        if (threadIdx.x == 0) RD_PF_TRACE(1, 47, b >> 1);
      }
      if (gt == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // shared memory outlives the copies
    }
  }
  if (aborted && threadIdx.x == 0)   // whatever is still under way lands first
    for (const unsigned long long t0 = global_ns(); global_ns() - t0 < 1000000ull;) {}
  tc_fence_before();
  cluster_sync();   // the pair frees its tensor memory together
  if (threadIdx.x == 0) RD_PF_TRACE(0, 47, 5);   // epilogue stores done
  if (warp == 9) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols)
                 : "memory");
  }
}

// Combines the key-split records of a row: one warp-pair (64 threads, 4 dims each) per row
// (token, head); out = sum_z acc_z e^(m_z - M) / sum_z l_z e^(m_z - M), times sigmoid(gate)
// if given (the gate is only read). Rows whose records are all empty give zeros.
template <int kMax>   // records of a row at most
__global__ void __launch_bounds__(256)
prefill_merge_kernel(const float4 *__restrict__ rec_acc, const float2 *__restrict__ rec_ml, float *__restrict__ out,
                     const float *__restrict__ gate, int64_t n_rows, int n_splits) {
  const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 6);
  const int tx = threadIdx.x & 63;
  pdl_launch_dependents();
  pdl_wait();   // launched under the tile kernel: its records are complete from here on
  if (row >= n_rows) return;
  // every load of the row is requested before the first is used (at most kMax
  // records): one round trip to L2 instead of one for the maxima and one per record
  float m[kMax], lz[kMax];
  float4 va[kMax];
#pragma unroll
  for (int z = 0; z < kMax; ++z) {
    m[z] = -INFINITY;
    lz[z] = 0.f;
    va[z] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (z < n_splits) {
      const float2 ml = __ldcg(rec_ml + row * n_splits + z);
      m[z] = ml.x;
      lz[z] = ml.y;
      va[z] = __ldcg(rec_acc + (row * n_splits + z) * (kHeadDim / 4) + tx);
    }
  }
  float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
  if (gate != nullptr) g = *reinterpret_cast<const float4 *>(gate + (size_t)row * kHeadDim + 4 * tx);
  float mm = -INFINITY;
#pragma unroll
  for (int z = 0; z < kMax; ++z) mm = fmaxf(mm, m[z]);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float l = 0.f;
  if (mm != -INFINITY) {
#pragma unroll
    for (int z = 0; z < kMax; ++z) {
      if (m[z] == -INFINITY) continue;
      const float w = __expf(m[z] - mm);
      l = fmaf(lz[z], w, l);
      acc.x = fmaf(va[z].x, w, acc.x);
      acc.y = fmaf(va[z].y, w, acc.y);
      acc.z = fmaf(va[z].z, w, acc.z);
      acc.w = fmaf(va[z].w, w, acc.w);
    }
  }
  const float inv = l > 0.f ? 1.0f / l : 0.f;
  float4 o = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
  if (gate != nullptr) {
    o.x *= __fdividef(1.0f, 1.0f + __expf(-g.x));
    o.y *= __fdividef(1.0f, 1.0f + __expf(-g.y));
    o.z *= __fdividef(1.0f, 1.0f + __expf(-g.z));
    o.w *= __fdividef(1.0f, 1.0f + __expf(-g.w));
  }
  *reinterpret_cast<float4 *>(out + (size_t)row * kHeadDim + 4 * tx) = o;
}

// Fused append: one block per token, a warp per K or V row. The K rows are rotated with the operation
// order of kv_append_kernel, both are rounded to f16 -- the bytes rd_kv_append stores for f16
// caches. The tile kernel is launched under it as a programmatic dependent launch. (Its blocks could fetch the query and
// gate rows to L2 while the tile kernel before them still runs; where they did, that kernel's own queries came
// later: 512 tokens at 0 360.8 -> 353.4 us without it, at 7680 1726 -> 1705, 16 layers.)
__global__ void __launch_bounds__(256)
kv_prep_kernel(const int32_t *__restrict__ pos, int n_rot, const float *__restrict__ k_new,
               const float *__restrict__ v_new, uint4 *__restrict__ k_dst, uint4 *__restrict__ v_dst, int nkv,
               const __grid_constant__ RopeTable tab, unsigned *flags, int n_flags) {
  __shared__ float2 s_cs[32];
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the wait comes first: the tile kernel reads what earlier kernels wrote without waiting for this one
  pdl_wait();
  pdl_launch_dependents();
  if (t == 0 && (int)threadIdx.x < n_flags) flags[threadIdx.x] = 0;   // (of a balanced tile launch)
  const bool is_k = warp < nkv;
  const size_t row = (size_t)t * nkv + (is_k ? warp : warp - nkv);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
  if (warp < 2 * nkv) {   // requested before the table is computed
    const float4 *src = reinterpret_cast<const float4 *>((is_k ? k_new : v_new) + row * kHeadDim);
    a = src[2 * lane];
    b = src[2 * lane + 1];
  }
  if ((int)threadIdx.x < n_rot / 2) {
    float c, s;
    sincosf((float)pos[t] * tab.f[threadIdx.x], &s, &c);
    s_cs[threadIdx.x] = make_float2(c, s);
  }
  __syncthreads();
  if (warp >= 2 * nkv) return;
  float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  if (is_k && n_rot > 0) {
    // lanes 0 .. n_rot / 8 - 1 hold the rotated dims; dims d and d + n_rot / 2 sit n_rot / 16 lanes apart
    const int half_lanes = n_rot / 16;
    const bool rot = lane < 2 * half_lanes, lo = lane < half_lanes;
    const int src = !rot ? lane : lo ? lane + half_lanes : lane - half_lanes;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float other = __shfl_sync(0xffffffffu, v[i], src);
      if (rot) {
        const float2 cs = s_cs[8 * (lo ? lane : lane - half_lanes) + i];
        v[i] = lo ? __fsub_rn(__fmul_rn(v[i], cs.x), __fmul_rn(other, cs.y))
                  : __fadd_rn(__fmul_rn(other, cs.y), __fmul_rn(v[i], cs.x));
      }
    }
  }
  (is_k ? k_dst : v_dst)[row * 32 + lane] =
      make_uint4(pack_h2(v[0], v[1]), pack_h2(v[2], v[3]), pack_h2(v[4], v[5]), pack_h2(v[6], v[7]));
}

// The key split of tiles of one head and 128 tokens: whether a call over f16 caches uses records at all, and how many
// rd_attn_prefill_typed has to have room for; what is launched is prefill_plan's choice below. A cost model of three
// constants: a key tile, a CTA's prologue + epilogue (the query tile is converted and the result written whatever the key
// count) and a record (written by the tile kernel, read by the merge pass) in the ratio 2 : 9 : 0.0005, those of the kernel
// before the pairs of CTAs. Splitting pays only when the waves it saves outweigh the fixed costs it multiplies: 512
// tokens x 24 heads gain from about 8192 keys upwards (3 splits: 96 -> 288 CTAs = two full waves of 148 SMs), shorter
// prefixes do not. Measured at commit 430ed0c, which launched this split, us a layer with gate and rotation, by split
// count (this rule's in brackets):
//   tokens of keys     1        2        3        4        5        6        7       8
//     24 of  4000    51.1     31.8     26.8    [23.7]    24.6     23.3     34.7    33.4
//     60 of  9000    98.8     56.7     45.2     39.1     35.0    [32.2]    52.0    49.2
//    130 of  4130    56.6     39.6    [33.2]    48.5     47.3     47.0     55.1    57.0
//    200 of 12000   133.4     80.1    [65.1]    92.0     81.1     76.7     97.5    92.6
//    389 of 12346   164.6    172.3   [135.1]   154.6    168.1    164.6    170.2   182.4
//    512 of  4096   [62.9]    76.9     68.6     86.1    102.8    104.3    121.5   139.4
//    512 of  8192   113.8    129.9    [99.4]   119.6    137.9    133.9    150.9   168.4
//    512 of 16384   220.3    224.5   [169.4]   210.4    242.3    214.7    218.9   239.0
//   1000 of  8192   211.7    215.1   [209.5]   251.9    260.2    271.5    297.8   320.5
//   2048 of  8192  [329.2]   404.1    420.4    456.4    505.8    535.3    589.2   618.2
int prefill_splits(int n_q, int keys_total, int n_head, int sms) {
  const int ctas = ((n_q + kPfM - 1) / kPfM) * n_head;
  const int tiles = (keys_total + kPfN - 1) / kPfN;
#ifdef RD_TIMING_SWITCHES
  if (const char *e = getenv("RD_PF_SPLITS")) {   // timing builds: force a split count
    const int z = atoi(e);
    if (z >= 1 && z <= kPfMaxSplits && z <= tiles) return z;
  }
#endif
  auto cost = [&](int z) {
    const double waves = (double)((ctas * z + sms - 1) / sms);
    return waves * ((double)tiles / z * 2.0 + 9.0) + (z > 1 ? 0.0005 * n_q * n_head * z : 0.0);
  };
  int best = 1;
  double best_cost = cost(1) * 0.92;   // a split must win clearly to be worth its records
  for (int z = 2; z <= 8 && tiles / z >= 8; ++z) {
    if (cost(z) < best_cost) {
      best_cost = cost(z);
      best = z;
    }
  }
  return best;
}
// The rows of a CTA and the key splits of a launch. In key tiles (1.05 us): a wave of CTAs takes its tiles and nine
// more (prologue and epilogue, 19800 cycles), a record of a row 0.00045 (written, and read by the merge launch).
// Three heads of 42 tokens leave fewer rows empty than one head of 128 where the tokens end soon behind a tile's
// edge or do not fill a tile, and their smaller launch leaves room for more key ranges. Where both cost the same, the
// smaller split launch is the faster one, of unsplit ones that with one head (its warps without a row do nothing).
// us a layer with the chunk's append, one head | three heads, best split in brackets (this table and the next: one GPU,
// one build, forms forced):
//     24 of 24024   59.3 (6) | 37.2 (18)       130 of  4130   35.3 (3) | 32.2 (4)       31 of   31   15.4 | 17.4
//     60 of  9060   34.2 (6) | 32.2 (8)        200 of 12200   64.2 (3) | 62.5 (3)      450 of 4450   62.2 | 60.5
//    700 of  5700   79.0     | 78.2            389 of 12346  124.7 (3) | 121.2 (3)    1500 of 4500  120.1 | 121.0
// A balanced launch has no empty SMs in its last wave and a fifth of the records, combined where they are wanted
// instead of by a launch of their own; but most pairs of CTAs work on two parts, so it costs a run, the prologue (6) and
// epilogue of both (a record 4, the output 5.5) and 1.5 per record read. It has to win by 5 %: long passes run at
// the power cap, where idle SMs leave the others a higher clock. Best of the other two forms | balanced with one head |
// with three:
//    389 of 12346  121.2 | 121.7 | 112.8      450 of 9450   103.6 |  99.8 | 102.5    1000 of 8000   185.3 | 161.3 | 163.6
//    512 of 12512  133.7 | 125.9 | 143.2      512 of 8192    98.7 |  91.5 |  96.6     640 of 9640   118.7 | 121.0 | 128.7
//    260 of 12260   82.8 |  98.3 |  91.0      200 of 12200   62.5 |  77.8 |  75.3     700 of 5700    78.2 |  92.8 |  90.5
PrefillPlan prefill_plan(int n_q, int keys_total, int n_head, int sms, size_t record_bytes) {
  PrefillPlan best = {1, 1, 0};
  const int tiles = (keys_total + kPfN - 1) / kPfN;
#ifdef RD_TIMING_SWITCHES
  if (const char *e = getenv("RD_PF_FORM")) {   // timing builds: force heads and splits
    best.heads = atoi(e);
    if (const char *f = getenv("RD_PF_SPLITS")) best.splits = atoi(f);
    if (const char *f = getenv("RD_PF_PAIRS")) best.pairs = atoi(f);
    return best;
  }
#endif
  auto cost = [&](int heads, int z) {
    const int ctas = (n_q + pf_tokens(heads) - 1) / pf_tokens(heads) * (n_head / heads) * z;
    return (double)((ctas + sms - 1) / sms) * ((double)tiles / z + 9.0) + (z > 1 ? 0.00045 * n_q * n_head * z : 0.0) +
           (heads == 3 && z > 1 ? -0.01 : 0.0);
  };
  double best_cost = cost(1, 1);
  for (int heads = 1; heads <= 3; heads += 2)
    for (int z = 1; z <= kPfMaxSplits && (z == 1 || tiles / z >= 4); ++z) {
      if (prefill_record_bytes(n_q, n_head, z) > record_bytes) break;
      if (cost(heads, z) < best_cost) {
        best_cost = cost(heads, z);
        best = {heads, z, 0};
      }
    }
  PrefillPlan balanced = {1, 1, 0};
  double balanced_cost = 0.0;
  for (int heads = 1; heads <= 3; heads += 2) {
    const int units = (n_q + pf_tokens(heads) - 1) / pf_tokens(heads) * (n_head / heads / 2);
    if (keys_total < n_q || tiles > 60000) continue;
    int pairs = sms / 2 < 120 ? sms / 2 : 120;   // (240 flags, zeroed by one block)
    const size_t room = record_bytes / (2 * (kPfRecBytes + sizeof(unsigned)));
    if ((size_t)pairs > room) pairs = (int)room;
    if (pairs < 2 || units + pairs > kPfMaxParts) continue;
    int64_t all = 0;
    for (int t = 0; t * pf_tokens(heads) < n_q; ++t)
      all += (int64_t)(n_head / heads / 2) * pf_unit_tiles(t, pf_tokens(heads), n_q, keys_total);
    if (all / pairs < 4) continue;
    const double run = (double)all / pairs, parts = tiles / run + 1;
    if (parts > kPfMaxRecords - 1) continue;
    const double c = run + 21.5 + 1.5 * tiles / run;
    if (c < 0.95 * best_cost && (balanced.pairs == 0 || c < balanced_cost)) {
      balanced_cost = c;
      balanced = {heads, 1, pairs};
    }
  }
  return balanced.pairs > 0 ? balanced : best;
}
int prefill_tile_tokens(int heads) { return pf_tokens(heads); }
size_t prefill_record_bytes(int n_q, int n_head, PrefillPlan plan) {
  return plan.pairs > 0 ? plan.pairs * 2 * (kPfRecBytes + sizeof(unsigned)) : prefill_record_bytes(n_q, n_head, plan.splits);
}
unsigned *prefill_flags(void *records, PrefillPlan plan) {
  return plan.pairs > 0 ? (unsigned *)((char *)records + plan.pairs * 2 * kPfRecBytes) : nullptr;
}
size_t prefill_record_bytes(int n_q, int n_head, int splits) {
  return splits > 1 ? (size_t)n_q * n_head * splits * kRec * sizeof(float) : 0;
}

// The parts of a balanced launch in the order of its grid; their number, or 0 if they do not fit.
static int balanced_parts(PrefillArgs::Part *out, int n_q, int keys, int groups, int tokens, int pairs) {
  const int tiles = (n_q + tokens - 1) / tokens, units = tiles * groups;
  int64_t all = 0;
  for (int t = 0; t < tiles; ++t) all += (int64_t)groups * pf_unit_tiles(t, tokens, n_q, keys);
  if (units + pairs > kPfMaxParts || all < pairs) return 0;
  PrefillArgs::Part rest[kPfMaxParts];
  int n_left = 0, n_rest = 0, run = 1;   // run: the next cut lies at all * run / pairs
  int64_t before = 0;                    // key tiles of the units before this one
  for (int unit = 0; unit < units; ++unit) {
    const int n = pf_unit_tiles(unit / groups, tokens, n_q, keys);
    PrefillArgs::Part first = {(unsigned short)unit, 0, (unsigned short)n, (unsigned short)n_left, 0};
    for (; all * run / pairs < before + n; ++run) {
      const int at = (int)(all * run / pairs - before);
      if (at == 0) continue;   // (a cut between two units)
      if (first.n_rec == 0) first.c1 = (unsigned short)at;
      else out[n_left - 1].c1 = (unsigned short)at;
      out[n_left] = {(unsigned short)unit, (unsigned short)at, (unsigned short)n, (unsigned short)n_left, 0};
      ++n_left;
      ++first.n_rec;
    }
    if (first.n_rec > kPfMaxRecords) return 0;
    before += n;
    rest[n_rest++] = first;
  }
  std::stable_sort(rest, rest + n_rest, [](const PrefillArgs::Part &x, const PrefillArgs::Part &y) {
    return x.c1 - x.c0 > y.c1 - y.c0;
  });
  for (int i = 0; i < n_rest; ++i) out[n_left + i] = rest[i];
  return n_left + n_rest;
}

int prefill_ctas(PrefillPlan plan, int n_q, int keys_total, int n_head) {
  const int tokens = pf_tokens(plan.heads);
  if (plan.pairs == 0) return (n_q + tokens - 1) / tokens * (n_head / plan.heads) * plan.splits;
  PrefillArgs::Part parts[kPfMaxParts];
  return 2 * balanced_parts(parts, n_q, keys_total, n_head / plan.heads / 2, tokens, plan.pairs);
}

int launch_prefill(const float *q, const void *k, const void *v, float *out, const float *gate,
                   const int32_t *pos, int n_q, int keys_total, int n_head, int n_head_kv, float scale,
                   int n_rot, float freq_base, DeviceStatus *status, float *records, PrefillPlan plan,
                   const float *k_new, const float *v_new, void *k_dst, void *v_dst, bool kv_pending,
                   cudaStream_t st) {
  PrefillArgs a;
  memset(&a, 0, sizeof(a));
  int rc = encode_f16_tmap(&a.tm_k, k, n_head_kv, keys_total, kPfKKeys);
  if (rc != RD_OK) return rc;
  rc = encode_f16_tmap(&a.tm_v, v, n_head_kv, keys_total, kPfN);
  if (rc != RD_OK) return rc;
  a.q = q;
  a.gate = gate;
  a.pos = pos;
  a.n_q = n_q;
  a.n_head = n_head;
  a.qscale = scale * 1.4426950408889634f;
  const int heads = plan.heads, tokens = pf_tokens(heads), n_splits = records == nullptr ? 1 : plan.splits;
  if (n_splits < 1 || n_splits > kPfMaxSplits || (heads != 1 && heads != 3)) return RD_ERR_SHAPE;
  int n_parts = 0;
  if (plan.pairs > 0) {
    if (records == nullptr || n_splits != 1) return RD_ERR_SHAPE;
    a.rec = (float4 *)records;
    a.flags = prefill_flags(records, plan);
    a.groups = n_head / heads / 2;
    a.keys = keys_total;
    n_parts = balanced_parts(a.parts, n_q, keys_total, a.groups, tokens, plan.pairs);
    if (n_parts <= 0) return RD_ERR_SHAPE;
  }
  if (n_splits > 1) {
    a.rec_ml = reinterpret_cast<float2 *>(records + (size_t)n_q * n_head * n_splits * kHeadDim);
    if ((rc = encode_f32_tmap(&a.tm_o, records, kHeadDim * n_splits, n_head, n_q, heads, tokens)) != RD_OK) return rc;
  } else {
    if (gate != nullptr && (rc = encode_f32_tmap(&a.tm_g, gate, kHeadDim, n_head, n_q, heads, tokens)) != RD_OK) return rc;
    if ((rc = encode_f32_tmap(&a.tm_o, out, kHeadDim, n_head, n_q, heads, tokens)) != RD_OK) return rc;
  }
  a.n_rot = n_rot;
  if (n_rot > 0) memcpy(a.freq, make_rope_table(n_rot, freq_base).f, sizeof(a.freq));
  a.kv_wait = k_new != nullptr || kv_pending ? 1 : 0;
  a.status = status;
  a.debug = 0;
#ifdef RD_TIMING_SWITCHES
  if (const char *e = getenv("RD_PREFILL_DEBUG")) a.debug = atoi(e);
#endif
  static bool attr_set[32] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return RD_ERR_CUDA;
  if (dev < 0 || dev >= 32 || !attr_set[dev]) {
    for (auto *f : {prefill_kernel<1, false>, prefill_kernel<3, false>, prefill_kernel<1, true>, prefill_kernel<3, true>})
      if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kPfSmemBytes) != cudaSuccess)
        return RD_ERR_CUDA;
    if (dev >= 0 && dev < 32) attr_set[dev] = true;
  }
  if (k_new != nullptr) {
    if (launch_pdl(8, kv_prep_kernel, dim3((unsigned)n_q), dim3(256), 0, st, pos, n_rot, k_new, v_new,
                   (uint4 *)k_dst, (uint4 *)v_dst, n_head_kv, make_rope_table(n_rot, freq_base), a.flags, 2 * plan.pairs) != cudaSuccess)
      return RD_ERR_CUDA;
  } else if (plan.pairs > 0 && !kv_pending) {   // (no launch of this call that zeroes the flags)
    if (cudaMemsetAsync(a.flags, 0, 2 * plan.pairs * sizeof(unsigned), st) != cudaSuccess) return RD_ERR_CUDA;
  }
  auto *kernel = plan.pairs > 0 ? (heads == 1 ? prefill_kernel<1, true> : prefill_kernel<3, true>)
                                : (heads == 1 ? prefill_kernel<1, false> : prefill_kernel<3, false>);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = plan.pairs > 0 ? dim3(2 * (unsigned)n_parts)
                               : dim3((unsigned)(n_head / heads), (unsigned)((n_q + tokens - 1) / tokens), (unsigned)n_splits);
  cfg.blockDim = dim3(kPfThreads);
  cfg.dynamicSmemBytes = kPfSmemBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;   // a pair must lie along x
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  // starts under the launch before it, see PrefillArgs::kv_wait
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, kernel, a) != cudaSuccess) return RD_ERR_CUDA;
  if (n_splits > 1) {
    const int64_t n_rows = (int64_t)n_q * n_head;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((n_rows + 3) / 4));
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, n_splits <= 8    ? prefill_merge_kernel<8>
                                 : n_splits <= 12 ? prefill_merge_kernel<12>
                                                  : prefill_merge_kernel<kPfMaxSplits>,
                           (const float4 *)records, (const float2 *)a.rec_ml, out,
                           gate, n_rows, n_splits) !=
        cudaSuccess)
      return RD_ERR_CUDA;
  }
  return RD_OK;
}

}  // namespace rd

#ifdef RD_PF_TRACING
extern "C" int rd_debug_pf_trace(unsigned long long *host_dst) {
  return cudaMemcpyFromSymbol(host_dst, g_pf_trace, sizeof(g_pf_trace)) == cudaSuccess ? 0 : -1;
}
#endif
