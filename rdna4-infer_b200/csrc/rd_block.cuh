// Attention of a BLOCK of query tokens (speculative verify, short chunks) over caches of any type:
// up to eight tokens share every dequantized K and V value.
//
// Replaces attn_batch_kernel / attn_split_batch_kernel (include/rdna4/attn.cuh:268-424, 686-1049),
// which re-read and re-expand the prefix for every token. Grid (n_splits, n_head_kv, token chunks) or
// (work items, n_head_kv): a CTA owns a run of 64-key slots of one KV head and the 6 T <= 48 score
// columns (token, query head) of its chunk, NT = 2, 3, 4 or 6 MMA tiles of 8 columns.
//
// The CTA's warps form teams of four; a team streams slots through its own ring with 16-byte
// asynchronous copies, every warp 16 of the 64 rows. Per slot
//   * warp w multiplies keys 16 w .. 16 w + 15, the K rows it has copied itself, with all columns (K
//     fragments dequantized in registers once, query fragments from shared memory), and requests
//     its K rows of a later slot;
//   * one barrier (with the vote "does any score exceed the team's reference?") frees the previous
//     V slot, into which the warps request their V rows of a later one;
//   * the weights go to shared memory as MMA fragments, a second barrier publishes them and the V
//     rows, and warp w multiplies all 64 keys with its quarter of the output dims: every V value is
//     dequantized once, by one warp, and a warp holds 16 NT accumulators where a warp with all dims
//     would hold 64 NT.
// The columns of a slot share its V rows, also those behind the last key of a column's own token, with weight
// 0. A non-finite value there (an f16 cache saturates to infinity) would make that 0 a NaN, so a launch whose
// accumulators are not all finite runs the key loop once more, token by token (careful_pv). Any other launch pays
// one check of its accumulators for that.
// Precision: the weight of the key that is the reference is exactly 1 in f16, the others are rounded, and a reference
// per team leaves fewer exact ones than one per 16 keys. The weights of a team's first slot therefore go to the tensor
// cores in two f16 parts (a second pass of P V over the same slot), which makes up for it where the runs
// are short; long runs never had much of it. Error against 64 bits, f16, with one reference per 16 keys / without the
// second part / with it: 2 tokens over 100 keys 2.36 / 2.75 / 1.93e-4, 5 over 4096 2.87 / 2.97 / 2.52e-4, 5 over 20011
// 2.94 / 2.96 / 2.87e-4. It costs 1.2 us a launch: 5 tokens over 20011 q4_0 keys 463 -> 483 us for 16 layers.
// (Both parts for every slot: 511 us, 2.11e-4.)
// (Tensor-map boxes of one head's rows were the slower copy: the TMA unit fetches whole cache lines,
// and a 272-byte row of q8_0 lies in three of them. 64 sequences of 1024 to 32768 keys
// verifying four tokens: copies alone 817 us.)
// One record (m, l, acc[256]) per (token, head) and split, merged by merge_kernel.
//
// What bounds it: latency. Two or three warps per scheduler (registers), each a chain of shared-memory loads,
// dequantization, mma.sync, vote, exponentials, fragment stores, barrier, mma.sync (with two: issue in 35 % of the active
// cycles, tensor pipe 22 %, DRAM 12 % over 20011 q4_0 keys). Of the 33000 cycles of a CTA there (5 tokens, two teams, behind
// the wait for the launch before it) 7800 lie before the first slot, 7800 in it (references, the second part of its weights,
// cold code), 13200 in the others, 4200 in the records; with three teams 7800, 10200, 9000 and 5400.
// A third team, where rings and registers allow it, pays where runs are long (launch_block_tiles); the query rows are
// requested first and converted under the first slot's copies, since a whole ring's copies take 4400 cycles to issue.
//   us a layer with its pre-attention, merge and gate launches, commit 430ed0c (two teams, ring first, records by two dims a
//   thread, merge of eight records at a time) | now (two teams; many sequences, without those launches, three):
//                        5000 keys     20011 keys    32 sequences of 4096 to 16384
//   q4_0, 5 tokens       22.5 | 20.1   31.5 | 28.1   319.7 | 292.1
//   q8_0, 4              22.3 | 19.8   31.4 | 28.0   302.3 | 290.0
//   q8_0/f16, 4          21.6 | 19.6   30.5 | 28.1   298.2 | 271.6
//   q5_0/q4_1, 5         23.3 | 21.2   33.1 | 29.6   330.0 | 312.5
//   f16, 4               22.8 | 19.4   34.5 | 31.0   (one team: two want 1 KB more than there is)
#pragma once
#include <string.h>

#include <type_traits>

#include "rd_frag.cuh"
#include "rd_internal.h"

namespace rd {

constexpr int kBlkKeys = 64;       // keys per slot
constexpr int kBlkSmem = 222 * 1024;   // dynamic; the static arrays take up to 4.5 KB
constexpr int kBlkQPair = 576;     // bytes of a pair of MMAs in a tile's query fragments: 512, shifted by half the banks
constexpr int kBlkPlane = 268;     // floats per column in the epilogue planes (12 mod 32)
constexpr float kBlkSlack = 8.0f;  // see kRefSlack
constexpr float kBlkNone = -1.0e30f;

// Column tiles for a chunk of n tokens: the smallest of the four forms that holds them. Six tokens have no form of
// their own (36 columns in 48); one of five tiles takes 23.5 instead of 26.1 us over 20011 q4_0 keys and is not built.
__host__ __device__ constexpr int block_tiles(int n) { return n <= 2 ? 2 : n <= 4 ? 3 : n == 5 ? 4 : 6; }

template <int KT, int VT, int NT, int MOST>
struct BlockGeo {
  static constexpr int kPK = slot_pitch(KT), kPV = slot_pitch(VT);
  static constexpr int kSK = kBlkKeys * kPK, kSV = kBlkKeys * kPV;   // multiples of 128
  static constexpr int kQBytes = NT * 8 * kBlkQPair;                          // query fragments
  static constexpr int kPBytes = NT * 2048;                          // weight fragments of a slot, two parts, per team
  static constexpr int kHead = 512 + kQBytes;                        // dim table, query fragments
  static constexpr int budget(int teams) { return (kBlkSmem - kHead) / teams - kPBytes; }
  // Teams, MOST at most (launch_block_tiles): three where each gets one slot and 168 registers hold its sums (up to four
  // column tiles), two where each gets one and another K or V of the next
  static constexpr int kPlaneBytes = NT * 8 * kBlkPlane * 4;   // a team's ring doubles as its plane
  static constexpr int kTeams = MOST >= 3 && NT <= 4 && budget(3) >= kSK + kSV && budget(3) >= kPlaneBytes   ? 3
                                : budget(2) >= kSK + kSV + (kSK < kSV ? kSK : kSV) ? 2
                                                                                   : 1;
  static constexpr int kRing = budget(kTeams) & ~127;
  static constexpr int kBoth = min_i(4, kRing / (kSK + kSV));
  // what is left takes one more V (K is refilled half a slot earlier than V)
  static constexpr int DK = kBoth, DV = kBoth < 4 && kRing >= kBoth * (kSK + kSV) + kSV ? kBoth + 1 : kBoth;
  static constexpr int kRingBytes = DK * kSK + DV * kSV;
  static constexpr int kTeamBytes = kPBytes + (kRingBytes > kPlaneBytes ? kRingBytes : (kPlaneBytes + 127) & ~127);
  static constexpr int kSmem = kHead + kTeams * kTeamBytes;
  static constexpr int kThreads = kTeams * 128;
  static_assert(kBoth >= 1 && kSK % 128 == 0 && kSV % 128 == 0 && kSmem <= kBlkSmem, "ring geometry");
};

struct BlockArgs {
  const float *q;                 // [n_tok][n_head][256]
  const uint8_t *k;
  const uint8_t *v;
  float *partial;                 // [n_tok][n_head][n_splits][258]
  const int32_t *pos;             // device: token i attends keys 0..pos[i]
  int n_tok;
  int chunk;                      // tokens per chunk
  int n_head;
  int nkv;
  float qscale;                   // scale * log2(e)
  const DecodeSeq *seqs;          // many sequences: CTA x works on items[x] = (sequence, first token, split)
  const int4 *items;
};

// Barrier of one team, and one that also ORs a predicate over it.
__device__ __forceinline__ void team_sync(int team) {
  asm volatile("bar.sync %0, 128;" ::"r"(1 + team) : "memory");
}
__device__ __forceinline__ bool team_any(int team, bool x) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)x), "r"(1 + team)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ void st_frag(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
// The keys 2 tq, 2 tq + 1, 2 tq + 8 and 2 tq + 9 behind `first` that are at most t: masks of an A fragment's halves.
__device__ __forceinline__ uint2 key_mask(int first, int t) {
  const uint32_t lo = (first <= t ? 0xffffu : 0u) | (first + 1 <= t ? 0xffff0000u : 0u);
  const uint32_t hi = (first + 8 <= t ? 0xffffu : 0u) | (first + 9 <= t ? 0xffff0000u : 0u);
  return make_uint2(lo, hi);
}
// O += V^T P^T of 16 keys (from key0 on) and one M-tile, every token with its own keys only: rows behind its last
// key count as zeros, and of a product only the token's six columns are taken.
template <int NT>
__device__ __forceinline__ void careful_pv(float (&O)[NT][4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        const uint2 (&pb)[NT], const int *s_t, int n_tok, int key0, int tq) {
#pragma unroll 1
  for (int j = 0; j < n_tok; ++j) {
    const uint2 mask = key_mask(key0 + 2 * tq, s_t[kGroup * j]);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (kGroup * j + kGroup <= 8 * nt || kGroup * j >= 8 * nt + 8) continue;   // no column of this token
      float x[4] = {0.f, 0.f, 0.f, 0.f};
      mma16816(x, a0 & mask.x, a1 & mask.x, a2 & mask.y, a3 & mask.y, pb[nt].x, pb[nt].y);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 8 * nt + 2 * tq + (e & 1);
        if (c >= kGroup * j && c < kGroup * j + kGroup) O[nt][e] += x[e];
      }
    }
  }
}

template <int KT, int VT, int NT, int MOST>
__global__ void __launch_bounds__(BlockGeo<KT, VT, NT, MOST>::kThreads, 1)
block_kernel(const __grid_constant__ BlockArgs p) {
  using Geo = BlockGeo<KT, VT, NT, MOST>;
  using KL = KLoad<KT>;
  using VL = VLoad<VT>;
  constexpr int RK = row_bytes(KT), RV = row_bytes(VT), PK = Geo::kPK, PV = Geo::kPV, SK = Geo::kSK, SV = Geo::kSV;
  constexpr int DK = Geo::DK, DV = Geo::DV, TEAMS = Geo::kTeams, COLS = NT * 8;
  // copies go out in the order K0 V0 K1 V1 ...; with a V slot more than K slots, V runs level with K
  constexpr int WAIT_K = DV > DK ? 2 * DK - 1 : 2 * DK - 2, WAIT_V = DV > DK ? 2 * DK : 2 * DK - 2;
  constexpr unsigned FULL = 0xffffffffu;

  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ int s_t[COLS];                                  // last key of the column's token (-1: padding)
  __shared__ float s_max[TEAMS][4][COLS], s_sum[TEAMS][4][COLS], s_ref[TEAMS][COLS];
  __shared__ float s_wt[TEAMS][COLS], s_ml[COLS][2];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tq = lane & 3;
  const int team = warp >> 2, part = warp & 3;
  const int kvh = blockIdx.y, nkv = p.nkv;
  const uint32_t sbase = smem_u32(smem);
  unsigned short *inv = reinterpret_cast<unsigned short *>(smem);
  const uint32_t qfrag = sbase + 512;
  const uint32_t team0 = sbase + Geo::kHead + team * Geo::kTeamBytes;
  const uint32_t ring_k = team0, ring_v = ring_k + DK * SK;
  const uint32_t pfrag = team0 + (Geo::kTeamBytes - Geo::kPBytes);

  // dim -> byte offset of the half in a column's query fragments (inverts KL::dim): 16 bytes per
  // (pair of MMAs, quad lane)
  for (int i = threadIdx.x; i < 256; i += Geo::kThreads) {
    const int tq_i = i >> 6, n_i = (i >> 2) & 15, e_i = i & 3;
    inv[KL::dim(tq_i, n_i, e_i)] =
        (unsigned short)((n_i >> 1) * kBlkQPair + tq_i * 16 + (n_i & 1) * 8 + (e_i >> 1) * 4 + (e_i & 1) * 2);
  }
  __syncthreads();
  pdl_wait();   // everything below reads what earlier kernels of the stream wrote

  int s, S, tok0, n_tok;
  const float *qsrc;
  const uint8_t *khead, *vhead;
  float *rec0;
  int t_seq = 0;
  if (p.items != nullptr) {
    const int4 item = p.items[blockIdx.x];
    if (item.x < 0) return;   // padding of a plan with a fixed item count
    const DecodeSeq &d = p.seqs[item.x];
    tok0 = item.y;
    s = item.z;
    S = d.n_splits;
    t_seq = d.t - (p.n_tok - 1);   // the first token's last key
    qsrc = d.q;
    khead = d.k;
    vhead = d.v;
    rec0 = p.partial + (size_t)d.rec_base * kRec;
  } else {
    tok0 = blockIdx.z * p.chunk;
    s = blockIdx.x;
    S = gridDim.x;
    qsrc = p.q;
    khead = p.k;
    vhead = p.v;
    rec0 = p.partial;
  }
  n_tok = min(p.chunk, p.n_tok - tok0);
  khead += (size_t)kvh * RK;
  vhead += (size_t)kvh * RV;
  const size_t kb = (size_t)nkv * RK, vb = (size_t)nkv * RV;
  // the query rows: requested before anything else, so that they do not queue behind the first slots
  constexpr int NQ = (COLS * 64 + Geo::kThreads - 1) / Geo::kThreads;
  float4 qv[NQ];
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    const int i = threadIdx.x + k * Geo::kThreads, c = i >> 6, j = c / kGroup, h = c % kGroup;
    qv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < COLS * 64 && j < n_tok)
      qv[k] = *reinterpret_cast<const float4 *>(qsrc + ((size_t)(tok0 + j) * p.n_head + kvh * kGroup + h) * kHeadDim +
                                                4 * (i & 63));
  }
  // last and first "last key" of the chunk's tokens
  int t_max = -1, t_min = 0x7fffffff;
  if (p.items != nullptr) {
    t_min = t_seq + tok0;
    t_max = t_min + n_tok - 1;
  } else {
    for (int i = 0; i < n_tok; ++i) {
      const int t = p.pos[tok0 + i];
      t_max = max(t_max, t);
      t_min = min(t_min, t);
    }
  }
  const int slots_total = (t_max + kBlkKeys) / kBlkKeys;   // ceil((t_max + 1) / 64)
  const int c_b = (int)(((int64_t)slots_total * s) / S), c_e = (int)(((int64_t)slots_total * (s + 1)) / S);
  // the team's slots: c_b + team + i * TEAMS
  const int n_mine = c_e - c_b > team ? (c_e - c_b - team + TEAMS - 1) / TEAMS : 0;

  // This warp's 16 rows of the team's i-th slot; always one commit group, empty behind the end.
  auto fill_k = [&](int i) {
    if (i < n_mine)
      copy_slot<KT>(ring_k + (i % DK) * SK + 16 * part * PK, khead, kb, (c_b + team + i * TEAMS) * kBlkKeys + 16 * part,
                    t_max, lane);
    cp_async_commit();
  };
  auto fill_v = [&](int i) {
    if (i < n_mine)
      copy_slot<VT>(ring_v + (i % DV) * SV + 16 * part * PV, vhead, vb, (c_b + team + i * TEAMS) * kBlkKeys + 16 * part,
                    t_max, lane);
    cp_async_commit();
  };
  auto fill_ring = [&](int first, int end) {
#pragma unroll 1
    for (int i = first; i < end; ++i) {
      fill_k(i);
      if (i + 1 < DV) fill_v(i);
    }
  };
  // the first slot now, the others behind the query fragments: the copies of a whole ring take thousands of cycles to issue
  // (many sequences: other CTAs' copies are under way whenever these are not)
  const bool early = p.items != nullptr;
  fill_ring(0, early ? DK : 1);

  for (int c = threadIdx.x; c < COLS; c += Geo::kThreads) {
    const int j = c / kGroup;
    s_t[c] = j < n_tok ? (p.items != nullptr ? t_seq + tok0 + j : p.pos[tok0 + j]) : -1;
  }
  // query fragments, pre-scaled into log2 units (and by the loader's fixed-point factor); the padding
  // columns are zero
  {
    const float qmul = p.qscale * KL::kUnscale;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const int i = threadIdx.x + k * Geo::kThreads, c = i >> 6;
      if (i >= COLS * 64) break;
      const uint32_t cb = qfrag + (c >> 3) * (8 * kBlkQPair) + (c & 7) * 64;
      const uint2 off = *reinterpret_cast<const uint2 *>(inv + 4 * (i & 63));
      const float x[4] = {qv[k].x, qv[k].y, qv[k].z, qv[k].w};
      const uint32_t o[4] = {off.x & 0xffffu, off.x >> 16, off.y & 0xffffu, off.y >> 16};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const unsigned short hbits = __half_as_ushort(__float2half_rn(x[e] * qmul));
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(cb + o[e]), "h"(hbits) : "memory");
      }
    }
  }
  if (!early) fill_ring(1, DK);
  __syncthreads();

  float O[4][NT][4];                     // [M-tile of this warp's quarter of the dims][column tile]
  float ref[NT][2], run[NT][2], l[NT][2];   // per lane column: team's reference, lane-local maximum and sum
  const uint32_t qlane = qfrag + lane * 16;
  bool careful = false;
#pragma unroll 1
  for (;;) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      ref[nt][0] = ref[nt][1] = run[nt][0] = run[nt][1] = kBlkNone;
      l[nt][0] = l[nt][1] = 0.f;
#pragma unroll
      for (int m = 0; m < 4; ++m) O[m][nt][0] = O[m][nt][1] = O[m][nt][2] = O[m][nt][3] = 0.f;
    }
#pragma unroll 1
    for (int i = 0; i < n_mine; ++i) {
      const int row0 = (c_b + team + i * TEAMS) * kBlkKeys;
      const bool fine = i == 0 && !careful;   // weights in two parts
      cp_async_wait<WAIT_K>();
      __syncwarp();
      // ---- S = K Q^T: this warp's 16 keys x all columns ----
      float Sv[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) Sv[nt][0] = Sv[nt][1] = Sv[nt][2] = Sv[nt][3] = 0.f;
      {
        const uint32_t kr = ring_k + (i % DK) * SK + (16 * part + g) * PK;
        uint4 qf[NT];
        KL::run(kr, kr + 8 * PK, tq, [&](int n, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            if ((n & 1) == 0) qf[nt] = lds128(qlane + nt * (8 * kBlkQPair) + (n >> 1) * kBlkQPair);
            mma16816(Sv[nt], a0, a1, a2, a3, (n & 1) ? qf[nt].z : qf[nt].x, (n & 1) ? qf[nt].w : qf[nt].y);
          }
        });
      }
      __syncwarp();
      fill_k(i + DK);
      if (row0 + kBlkKeys - 1 > t_min) {   // some column ends inside or before this slot
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (row0 + 16 * part + g + (e >> 1) * 8 > s_t[8 * nt + 2 * tq + (e & 1)]) Sv[nt][e] = -INFINITY;
      }
      bool grow = false;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          run[nt][e] = fmaxf(run[nt][e], fmaxf(Sv[nt][e], Sv[nt][e + 2]));
          grow |= run[nt][e] > ref[nt][e] + kBlkSlack;
        }
      // every warp of the team is done with the V slot before this one
      const bool any = team_any(team, grow);
      fill_v(i - 1 + DV);
      if (any) {
        // the team's references move to the current maxima of the columns (over its 64 key rows)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float m = run[nt][e];
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
            if (g == 0) s_max[team][part][8 * nt + 2 * tq + e] = m;
          }
        team_sync(team);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int c = 8 * nt + 2 * tq + e;
            const float m = fmaxf(fmaxf(fmaxf(s_max[team][0][c], s_max[team][1][c]),
                                        fmaxf(s_max[team][2][c], s_max[team][3][c])), ref[nt][e]);
            const float f = ex2(ref[nt][e] - m);
            ref[nt][e] = m;
            l[nt][e] *= f;
#pragma unroll
            for (int mt = 0; mt < 4; ++mt) {
              O[mt][nt][e] *= f;
              O[mt][nt][e + 2] *= f;
            }
          }
      }
      // ---- P^T fragments of this warp's keys -> shared memory ----
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const float p0 = ex2(Sv[nt][0] - ref[nt][0]), p1 = ex2(Sv[nt][1] - ref[nt][1]);
        const float p2 = ex2(Sv[nt][2] - ref[nt][0]), p3 = ex2(Sv[nt][3] - ref[nt][1]);
        const uint32_t h01 = pack_h2(p0, p1), h23 = pack_h2(p2, p3);
        const float2 r01 = unpack_h2(h01), r23 = unpack_h2(h23);
        const uint32_t at = pfrag + (part * NT + nt) * 256 + lane * 8;
        st_frag(at, movmatrix_trans(h01), movmatrix_trans(h23));
        if (fine) {
          st_frag(at + NT * 1024, movmatrix_trans(pack_h2(p0 - r01.x, p1 - r01.y)),
                  movmatrix_trans(pack_h2(p2 - r23.x, p3 - r23.y)));
          l[nt][0] += p0 + p2;
          l[nt][1] += p1 + p3;
        } else {   // the sums take the weights as rounded: a common rounding error of a column cancels in the quotient
          l[nt][0] += r01.x + r23.x;
          l[nt][1] += r01.y + r23.y;
        }
      }
      cp_async_wait<WAIT_V>();
      team_sync(team);
      // ---- O^T += V^T P^T: 64 keys x this warp's quarter of the dims ----
      auto pv = [&](int ks, uint32_t frag, auto &&mma) {
        uint2 pb[NT];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) pb[nt] = lds64(frag + (ks * NT + nt) * 256 + lane * 8);
        const uint32_t r0 = ring_v + (i % DV) * SV + (16 * ks + 2 * tq) * PV;
        const uint32_t rows[4] = {r0, r0 + PV, r0 + 8 * PV, r0 + 9 * PV};
        VL::run_part(rows, g, part, [&](int m, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
          mma(m, a0, a1, a2, a3, pb);
        });
      };
      if (!careful) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          pv(ks, pfrag, [&](int m, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, const uint2(&pb)[NT]) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma16816(O[m][nt], a0, a1, a2, a3, pb[nt].x, pb[nt].y);
          });
        if (fine) {
#pragma unroll 1
          for (int ks = 0; ks < 4; ++ks)
            pv(ks, pfrag + NT * 1024, [&](int m, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, const uint2(&pb)[NT]) {
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) mma16816(O[m][nt], a0, a1, a2, a3, pb[nt].x, pb[nt].y);
            });
        }
      } else {
#pragma unroll 1
        for (int ks = 0; ks < 4; ++ks)
          pv(ks, pfrag, [&](int m, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, const uint2(&pb)[NT]) {
            careful_pv<NT>(O[m], a0, a1, a2, a3, pb, s_t, n_tok, row0 + 16 * ks, tq);
          });
      }
    }
    cp_async_wait<0>();   // (only empty groups are left)
    float finite = 0.f;   // 0, or NaN where an accumulator is not finite
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) finite = fmaf(O[m][nt][e], 0.f, finite);
    // (also frees the rings)
    if (!__syncthreads_or(!careful && finite != 0.f)) break;
    careful = true;
    fill_ring(0, DK);
  }

  // ---- the teams meet ----
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float m = run[nt][e], ll = l[nt][e];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
        ll += __shfl_xor_sync(FULL, ll, o);
      }
      if (g == 0) {
        const int c = 8 * nt + 2 * tq + e;
        s_max[team][part][c] = m;
        s_sum[team][part][c] = ll;
        if (part == 0) s_ref[team][c] = ref[nt][e];
      }
    }
  // accumulators into the team's plane [column][dim] over its ring: dim d at 33 * (d >> 5) + (d & 31)
  {
    float *plane = reinterpret_cast<float *>(smem + Geo::kHead + team * Geo::kTeamBytes);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int d0 = VL::dim(g, 4 * part + m, 0), d1 = VL::dim(g, 4 * part + m, 1);
      const int a0 = 33 * (d0 >> 5) + (d0 & 31), a1 = 33 * (d1 >> 5) + (d1 & 31);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        float *pc = plane + (8 * nt + 2 * tq) * kBlkPlane;
        pc[a0] = O[m][nt][0];
        pc[a0 + kBlkPlane] = O[m][nt][1];
        pc[a1] = O[m][nt][2];
        pc[a1 + kBlkPlane] = O[m][nt][3];
      }
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < n_tok * kGroup; c += Geo::kThreads) {
    float mm = kBlkNone, ll = 0.f;
#pragma unroll
    for (int i = 0; i < TEAMS * 4; ++i) mm = fmaxf(mm, s_max[i >> 2][i & 3][c]);
    const bool empty = mm <= 0.5f * kBlkNone;
#pragma unroll
    for (int i = 0; i < TEAMS; ++i) {
      const float w = ex2(s_ref[i][c] - mm);   // references never exceed the true maximum
      s_wt[i][c] = empty ? 0.f : w * VL::kUnscale;
      ll = fmaf((s_sum[i][0][c] + s_sum[i][1][c]) + (s_sum[i][2][c] + s_sum[i][3][c]), w, ll);
    }
    s_ml[c][0] = empty ? -INFINITY : mm * 0.6931471805599453f;   // natural log
    s_ml[c][1] = empty ? 0.f : ll;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n_tok * kGroup * (kHeadDim / 4); i += Geo::kThreads) {   // four dims of a column
    const int c = i >> 6, dd = 4 * (i & 63);
    const int off = c * kBlkPlane + 33 * (dd >> 5) + (dd & 31);
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < TEAMS; ++w) {
      const float *pl = reinterpret_cast<const float *>(smem + Geo::kHead + w * Geo::kTeamBytes) + off;
      const float wt = s_wt[w][c];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = fmaf(pl[e], wt, a[e]);
    }
    float *rec = rec0 + (((size_t)(tok0 + c / kGroup) * p.n_head + kvh * kGroup + c % kGroup) * S + s) * kRec;
    if (dd == 0) {
      rec[0] = s_ml[c][0];
      rec[1] = s_ml[c][1];
    }
    if ((reinterpret_cast<uintptr_t>(rec) & 7) == 0) {   // always, for the library's workspace
      *reinterpret_cast<float2 *>(rec + 2 + dd) = make_float2(a[0], a[1]);
      *reinterpret_cast<float2 *>(rec + 4 + dd) = make_float2(a[2], a[3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) rec[2 + dd + e] = a[e];
    }
  }
}

template <int KT, int VT, int NT, int MOST>
int launch_block_teams(const BlockArgs &k, dim3 grid, cudaStream_t st) {
  using Geo = BlockGeo<KT, VT, NT, MOST>;
  static bool attr_set[32] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return RD_ERR_CUDA;
  if (dev < 0 || dev >= 32 || !attr_set[dev]) {
    if (cudaFuncSetAttribute(block_kernel<KT, VT, NT, MOST>, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo::kSmem) !=
        cudaSuccess)
      return RD_ERR_CUDA;
    if (dev >= 0 && dev < 32) attr_set[dev] = true;
  }
  return launch_pdl(2, block_kernel<KT, VT, NT, MOST>, grid, dim3(Geo::kThreads), Geo::kSmem, st, k) == cudaSuccess
             ? RD_OK
             : RD_ERR_CUDA;
}
// Two teams or three, by the 64-key slots of a CTA's run: `slots`, the mean over the items of many sequences (0: unknown,
// the key count of one sequence is on the device), and whether the CTAs make more than a wave.
// A third team shortens the run, but leaves each team a shallower ring (f16 values: one slot) and adds to the prologue and
// to the planes that meet at the end. Measured, speed against commit 430ed0c, three teams | two:
//   slots (items of a KV head)   8 (32)       16 (32)      24 (32)      24 (64)      32 (32)      34 (72)      64 (32)    147 (37)
//   q8_0/f16, 2 tokens           0.91 | 1.03  0.91 | 1.02  0.91 | 1.00  0.96 | 1.00  0.94 | 1.00  1.04 | 1.00  0.99 | 1.01  1.11 | 0.99
//   f16, 2                       0.95 | 1.01  0.94 | 1.00  0.95 | 1.00  1.00 | 1.02  0.96 | 1.00  1.06 | 1.00  0.99 | 1.00  1.11 | 1.00
//   q4_0, 3                      0.97 | 1.00  1.03 | 1.03  1.02 | 1.02  1.02 | 1.02  1.02 | 1.02  1.03 | 1.00
//   q5_0/q4_1, 4                 1.03 | 1.03  1.08 | 1.02  1.08 | 1.02  1.06 | 1.02  1.09 | 1.03  1.10 | 1.03
// One sequence, 4 tokens         500 keys      5000          20011         40000
//   q8_0/f16                     1.06 | 1.13   1.03 | 1.10   1.01 | 1.10   1.01 | 1.07
//   q4_0                         1.06 | 1.13   1.08 | 1.11   1.04 | 1.10   1.06 | 1.07
//   q5_0/q4_1                    1.12 | 1.12   1.08 | 1.08   1.16 | 1.14   1.14 | 1.09
// (37 CTAs a KV head: 40000 keys are 17 slots.)
struct BlockRuns {
  int slots;
  bool waves;
};
template <int KT, int VT, int NT>
int launch_block_tiles(const BlockArgs &k, dim3 grid, BlockRuns runs, cudaStream_t st) {
  using Three = BlockGeo<KT, VT, NT, 3>;
  if constexpr (Three::kTeams == 3) {
    if (runs.slots >= (Three::DK > 1 ? 16 : runs.waves ? 28 : 80)) return launch_block_teams<KT, VT, NT, 3>(k, grid, st);
  }
  return launch_block_teams<KT, VT, NT, 2>(k, grid, st);
}
template <int KT, int VT>
int launch_block_chunk(const BlockArgs &k, dim3 grid, BlockRuns runs, cudaStream_t st) {
  switch (block_tiles(k.chunk)) {
    case 2: return launch_block_tiles<KT, VT, 2>(k, grid, runs, st);
    case 3: return launch_block_tiles<KT, VT, 3>(k, grid, runs, st);
    case 4: return launch_block_tiles<KT, VT, 4>(k, grid, runs, st);
    default: return launch_block_tiles<KT, VT, 6>(k, grid, runs, st);
  }
}

// One sequence: grid (n_splits, n_head_kv, chunks of a.chunk tokens).
template <int KT, int VT>
int launch_block_typed(const DecodeArgs &a, int chunk, cudaStream_t st) {
  BlockArgs k;
  memset(&k, 0, sizeof(k));
  k.q = a.q;
  k.k = (const uint8_t *)a.k;
  k.v = (const uint8_t *)a.v;
  k.partial = a.partial;
  k.pos = a.pos;
  k.n_tok = a.n_tok;
  k.chunk = chunk;
  k.n_head = a.n_head;
  k.nkv = a.n_head_kv;
  k.qscale = a.scale * 1.4426950408889634f;
  return launch_block_chunk<KT, VT>(
      k, dim3((unsigned)a.n_splits, (unsigned)a.n_head_kv, (unsigned)((a.n_tok + chunk - 1) / chunk)), {0, false}, st);
}

// Many sequences: grid (work items, n_head_kv).
template <int KT, int VT>
int launch_block_multi_typed(const MultiDecodeArgs &a, cudaStream_t st) {
  BlockArgs k;
  memset(&k, 0, sizeof(k));
  k.partial = a.records;
  k.n_tok = a.q_len;
  k.chunk = block_chunk(a.q_len);
  k.n_head = a.n_head;
  k.nkv = a.n_head_kv;
  k.qscale = a.scale * 1.4426950408889634f;
  k.seqs = a.dev_seqs;
  k.items = a.dev_items;
  return launch_block_chunk<KT, VT>(k, dim3((unsigned)a.n_items, (unsigned)a.n_head_kv), {a.item_slots, a.waves}, st);
}

}  // namespace rd
