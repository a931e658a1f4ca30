// Fragment loaders of the decode-side attention kernels: stored K / V rows in shared memory,
// dequantized IN REGISTERS straight into mma.sync m16n8k16 f16 A fragments.
//
// Dequantization in two instructions per pair of values: masking a nibble (or
// placing a byte) into the low mantissa bits of a half gives the SUBNORMAL n * 2^-24
// exactly, and one HFMA2 with the block scale turns it into the value:
//   q4_0: fma(n * 2^-24, d * 2^12, -d * 2^-9)  = d * (n - 8)   * 2^-12
//   q8_0: fma(u * 2^-24, d * 2^12, -d * 2^-5)  = d * (u - 128) * 2^-12   (u = q ^ 0x80)
// rounded once, i.e. as exact as an f16 can hold the dequantized value. The common
// factor 2^-12 keeps every constant a power-of-two multiple of d inside the f16 range
// (block scales up to 16, i.e. |x| < 128 for q4_0) and is undone for free: Q is
// pre-multiplied by 2^12 for the scores, the output accumulator is multiplied by
// 2^12 once at the end.
//
// Index freedom used throughout: the contraction index of an MMA can be permuted
// freely as long as A and B agree, and the M index of P*V (the output dim) can be
// permuted freely as long as the epilogue writes each value to its true dim. Each
// loader below therefore defines `dim()` -- which true dim a fragment slot holds --
// and the Q fragments / epilogue are built from it.
#pragma once
#include "rd_common.cuh"

namespace rd {

constexpr uint32_t kH4096 = 0x6C006C00u;    // half2(2^12, 2^12)
constexpr uint32_t kH256 = 0x5C005C00u;     // half2(2^8, 2^8)
constexpr uint32_t kHNeg2m9 = 0x98009800u;  // half2(-2^-9, -2^-9)
constexpr uint32_t kHNeg2m5 = 0xA800A800u;  // half2(-2^-5, -2^-5)
constexpr float kQuantUnscale = 4096.0f;    // undoes the 2^-12 of the quantized loaders

// Per-block constants of the 4-bit path from the half2 scale d.
struct Q4Scale {
  uint32_t lo, hi, c;
  __device__ __forceinline__ explicit Q4Scale(uint32_t d)
      : lo(hmul2(d, kH4096)), hi(hmul2(d, kH256)), c(hmul2(d, kHNeg2m9)) {}
};
// q4_1: value = d*n + m (kv.h:219-229), same trick with the block minimum as the addend:
//   fma(n * 2^-24, d * 2^12, m * 2^-12) = (d*n + m) * 2^-12.
// (m * 2^-12 is a subnormal half for |m| < 1/4: at most 2^-13 of absolute error in the
// value, far inside the attention gates.)
constexpr uint32_t kH2m12 = 0x0C000C00u;    // half2(2^-12, 2^-12)
struct Q41Scale {
  uint32_t lo, hi, c;
  __device__ __forceinline__ Q41Scale(uint32_t d, uint32_t m)
      : lo(hmul2(d, kH4096)), hi(hmul2(d, kH256)), c(hmul2(m, kH2m12)) {}
};
// q5_0: value = d * ((nibble | bit5 << 4) - 16) (kv.h:203-216). The fifth bits of the four
// low-nibble and the four high-nibble elements of a word (bit i = byte i, bits above 7
// clear) are spread to bit 4 of each byte with one multiply -- bit i * 2^(4+7j) lands on
// 4+8j exactly for i == j and on positions the mask drops otherwise -- and OR-ed under the
// masked nibbles; the rest is the q4_0 trick with a 5-bit mantissa field:
//   fma(v * 2^-24, d * 2^12, -d * 2^-8) = d * (v - 16) * 2^-12.
constexpr uint32_t kHNeg2m8 = 0x9C009C00u;  // half2(-2^-8, -2^-8)
struct Q5Scale {
  uint32_t m, c;
  __device__ __forceinline__ explicit Q5Scale(uint32_t d) : m(hmul2(d, kH4096)), c(hmul2(d, kHNeg2m8)) {}
};
//   l0 = (B0.lo, B2.lo), h0 = (B0.hi, B2.hi), l1 = (B1.lo, B3.lo), h1 = (B1.hi, B3.hi)
__device__ __forceinline__ void dq5(uint32_t x, uint32_t bl, uint32_t bh, const Q5Scale &s, uint32_t &l0,
                                    uint32_t &h0, uint32_t &l1, uint32_t &h1) {
  const uint32_t xl = (x & 0x0F0F0F0Fu) | ((bl * 0x02040810u) & 0x10101010u);
  const uint32_t xh = ((x >> 4) & 0x0F0F0F0Fu) | ((bh * 0x02040810u) & 0x10101010u);
  l0 = hfma2(xl & 0x001F001Fu, s.m, s.c);
  l1 = hfma2((xl >> 8) & 0x001F001Fu, s.m, s.c);
  h0 = hfma2(xh & 0x001F001Fu, s.m, s.c);
  h1 = hfma2((xh >> 8) & 0x001F001Fu, s.m, s.c);
}
// One word of 8 nibbles, bytes (B0,B1,B2,B3) -> four half2 of d*(n-8)*2^-12 (Q4Scale) or
// (d*n+m)*2^-12 (Q41Scale):
//   l0 = (B0.lo, B2.lo), h0 = (B0.hi, B2.hi), l1 = (B1.lo, B3.lo), h1 = (B1.hi, B3.hi)
template <class Scale>
__device__ __forceinline__ void dq4(uint32_t x, const Scale &s, uint32_t &l0, uint32_t &h0,
                                    uint32_t &l1, uint32_t &h1) {
  const uint32_t y = x >> 8;
  l0 = hfma2(x & 0x000F000Fu, s.lo, s.c);
  h0 = hfma2(x & 0x00F000F0u, s.hi, s.c);
  l1 = hfma2(y & 0x000F000Fu, s.lo, s.c);
  h1 = hfma2(y & 0x00F000F0u, s.hi, s.c);
}
// Per-block constants of the 8-bit path.
struct Q8Scale {
  uint32_t m, c;
  __device__ __forceinline__ explicit Q8Scale(uint32_t d)
      : m(hmul2(d, kH4096)), c(hmul2(d, kHNeg2m5)) {}
};
// Four biased bytes u = q ^ 0x80: lo = (B0, B1), hi = (B2, B3), each d*q*2^-12.
__device__ __forceinline__ void dq8(uint32_t u, const Q8Scale &s, uint32_t &lo, uint32_t &hi) {
  lo = hfma2(prmt(u, 0u, 0x4140u), s.m, s.c);
  hi = hfma2(prmt(u, 0u, 0x4342u), s.m, s.c);
}

// Bytes between the rows of a slot that holds ONE head's rows in shared memory. Every loader below is
// free of bank conflicts when the pitch is 4 words mod 8: q8_0, q4_0 and q5_0 rows are already.
__host__ __device__ constexpr int slot_pitch(int type) {
  return row_bytes(type) + ((row_bytes(type) / 4) % 8 == 4 ? 0 : 16);
}
__host__ __device__ constexpr int min_i(int a, int b) { return a < b ? a : b; }

// =============================== copies ==========================================
__device__ __forceinline__ void cp_async16(uint32_t dst, const uint8_t *src) {
  asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One slot: rows row0 .. row0 + 15 of a head (`row_stride` bytes apart in the cache) to shared
// memory, kSlotKeys rows slot_pitch apart. Warp-collective; rows behind t_load are zeros (a weight of 0 times
// the last row again would be NaN where that row is infinite). Lanes are dealt so that a copy instruction takes whole rows: the lane's part of the address is a constant.
template <int T>
__device__ __forceinline__ void copy_slot(uint32_t dst, const uint8_t *head_base, size_t row_stride, int row0,
                                          int t_load, int lane) {
  constexpr int R = row_bytes(T), P = slot_pitch(T), CH = R / 16;
  // The ragged end: one slot of a launch, copies for the rows that exist and stores for the others (16 layers over
  // 137 f16 keys: 130 us; with a zero-filling copy per row 135, unrolled further 131 and 4096 keys 196 instead of 194).
  if (row0 + kSlotKeys - 1 > t_load) {
    const int have = t_load - row0 + 1 > 0 ? t_load - row0 + 1 : 0;   // rows that exist
#pragma unroll 2
    for (int i = lane; i < CH * have; i += 32)
      cp_async16(dst + (i / CH) * P + 16 * (i % CH), head_base + (size_t)(row0 + i / CH) * row_stride + 16 * (i % CH));
#pragma unroll 1
    for (int i = CH * have + lane; i < CH * kSlotKeys; i += 32)
      asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst + (i / CH) * P + 16 * (i % CH)), "r"(0) : "memory");
    return;
  }
  const uint8_t *src = head_base + (size_t)row0 * row_stride;
  if constexpr (CH == 17) {   // q8_0: two rows of 16 chunks per instruction, the 17th chunks in one
    const uint8_t *s0 = src + (size_t)(lane >> 4) * row_stride + 16 * (lane & 15);
    const uint32_t d0 = dst + (lane >> 4) * P + 16 * (lane & 15);
#pragma unroll
    for (int j = 0; j < 8; ++j) cp_async16(d0 + 2 * j * P, s0 + (size_t)(2 * j) * row_stride);
    if (lane < 16) cp_async16(dst + lane * P + 256, src + (size_t)lane * row_stride + 256);
  } else if constexpr (CH >= 32) {
#pragma unroll
    for (int j = 0; j < kSlotKeys; ++j)
#pragma unroll
      for (int c = 0; c < CH / 32; ++c)
        cp_async16(dst + j * P + 16 * (lane + 32 * c), src + (size_t)j * row_stride + 16 * (lane + 32 * c));
  } else {
    constexpr int RPI = 32 / CH;   // rows per instruction
    const int r = lane / CH, c = lane % CH;
    const uint8_t *s0 = src + (size_t)r * row_stride + 16 * c;
    const uint32_t d0 = dst + r * P + 16 * c;
#pragma unroll
    for (int j = 0; j < kSlotKeys; j += RPI)
      if (lane < RPI * CH && (j + RPI <= kSlotKeys || j + r < kSlotKeys))
        cp_async16(d0 + j * P, s0 + (size_t)j * row_stride);
  }
}

// =============================== K loaders =======================================
// A fragment of Q*K^T for MMA n (0..15): rows = keys g / g+8 of the 16-key group,
// k-slots (2t, 2t+1, 2t+8, 2t+9) = four dims chosen by the loader. run() calls
// mma(n, a0, a1, a2, a3) for n = 0..15. Values come out multiplied by 1/kUnscale.
template <int T>
struct KLoad;

template <>
struct KLoad<RD_KV_Q4_0> {
  static constexpr float kUnscale = kQuantUnscale;
  // lane t owns blocks 2t and 2t+1 of the row: 36 bytes at 36t (4-byte aligned).
  __device__ static int dim(int t, int n, int e) {
    const int x = n >> 1, odd = n & 1;
    int blk, i0, i2;
    if (x < 3) {
      blk = 2 * t; i0 = 4 * x + 2 + odd; i2 = i0 + 2;
    } else if (x == 3) {
      blk = 2 * t; i0 = odd; i2 = 14 + odd;
    } else {
      blk = 2 * t + 1; i0 = 4 * (x - 4) + odd; i2 = i0 + 2;
    }
    return blk * 32 + ((e & 1) ? i2 : i0) + ((e & 2) ? 16 : 0);
  }
  template <class F>
  __device__ static void run(uint32_t row_g, uint32_t row_h, int t, F &&mma) {
    uint32_t wg[9], wh[9];
    row_g += 36 * t;
    row_h += 36 * t;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      wg[i] = lds32(row_g + 4 * i);
      wh[i] = lds32(row_h + 4 * i);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const uint32_t dg = b == 0 ? prmt(wg[0], wg[0], 0x1010u) : prmt(wg[4], wg[4], 0x3232u);
      const uint32_t dh = b == 0 ? prmt(wh[0], wh[0], 0x1010u) : prmt(wh[4], wh[4], 0x3232u);
      const Q4Scale sg(dg), sh(dh);
#pragma unroll
      for (int xx = 0; xx < 4; ++xx) {
        const int x = 4 * b + xx;
        const uint32_t xg = (x == 3) ? prmt(wg[0], wg[4], 0x5432u) : wg[x + 1];
        const uint32_t xh = (x == 3) ? prmt(wh[0], wh[4], 0x5432u) : wh[x + 1];
        uint32_t l0g, h0g, l1g, h1g, l0h, h0h, l1h, h1h;
        dq4(xg, sg, l0g, h0g, l1g, h1g);
        dq4(xh, sh, l0h, h0h, l1h, h1h);
        mma(2 * x, l0g, l0h, h0g, h0h);
        mma(2 * x + 1, l1g, l1h, h1g, h1h);
      }
    }
  }
};

template <>
struct KLoad<RD_KV_Q8_0> {
  static constexpr float kUnscale = kQuantUnscale;
  // lane t owns blocks 2t and 2t+1: 68 bytes at 68t.
  __device__ static int dim(int t, int n, int e) {
    if (n < 7) return (2 * t) * 32 + 4 * n + 2 + e;
    if (n == 7) return (2 * t) * 32 + (e < 2 ? e : 28 + e);
    return (2 * t + 1) * 32 + 4 * (n - 8) + e;
  }
  template <class F>
  __device__ static void run(uint32_t row_g, uint32_t row_h, int t, F &&mma) {
    uint32_t wg[17], wh[17];
    row_g += 68 * t;
    row_h += 68 * t;
#pragma unroll
    for (int i = 0; i < 17; ++i) {
      wg[i] = lds32(row_g + 4 * i);
      wh[i] = lds32(row_h + 4 * i);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const uint32_t dg = b == 0 ? prmt(wg[0], wg[0], 0x1010u) : prmt(wg[8], wg[8], 0x3232u);
      const uint32_t dh = b == 0 ? prmt(wh[0], wh[0], 0x1010u) : prmt(wh[8], wh[8], 0x3232u);
      const Q8Scale sg(dg), sh(dh);
#pragma unroll
      for (int xx = 0; xx < 8; ++xx) {
        const int x = 8 * b + xx;
        uint32_t xg = (x == 7) ? prmt(wg[0], wg[8], 0x5432u) : wg[x + 1];
        uint32_t xh = (x == 7) ? prmt(wh[0], wh[8], 0x5432u) : wh[x + 1];
        xg ^= 0x80808080u;
        xh ^= 0x80808080u;
        uint32_t log_, hig, loh, hih;
        dq8(xg, sg, log_, hig);
        dq8(xh, sh, loh, hih);
        mma(x, log_, loh, hig, hih);
      }
    }
  }
};

template <>
struct KLoad<RD_KV_F16> {
  static constexpr float kUnscale = 1.0f;
  // lane t owns the 16-byte chunks 8*(i>>1) + 2t + (i&1), i = 0..7 (conflict-free with
  // a key pitch of 16 bytes mod 128).
  __device__ static int dim(int t, int n, int e) {
    const int i = n >> 1;
    const int c = 8 * (i >> 1) + 2 * t + (i & 1);
    return 8 * c + 4 * (n & 1) + e;
  }
  template <class F>
  __device__ static void run(uint32_t row_g, uint32_t row_h, int t, F &&mma) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = 8 * (i >> 1) + 2 * t + (i & 1);
      const uint4 vg = lds128(row_g + 16 * c);
      const uint4 vh = lds128(row_h + 16 * c);
      mma(2 * i, vg.x, vh.x, vg.y, vh.y);
      mma(2 * i + 1, vg.z, vh.z, vg.w, vh.w);
    }
  }
};

template <>
struct KLoad<RD_KV_F32> {
  static constexpr float kUnscale = 1.0f;
  // lane t owns the 16-byte chunks (4 dims) 4i + t, i = 0..15. Values are rounded to
  // f16 for the tensor core (f32 caches are a debugging format in the reference).
  __device__ static int dim(int t, int n, int e) { return 4 * (4 * n + t) + e; }
  template <class F>
  __device__ static void run(uint32_t row_g, uint32_t row_h, int t, F &&mma) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint4 vg = lds128(row_g + 16 * (4 * i + t));
      const uint4 vh = lds128(row_h + 16 * (4 * i + t));
      mma(i, pack_h2(__uint_as_float(vg.x), __uint_as_float(vg.y)),
          pack_h2(__uint_as_float(vh.x), __uint_as_float(vh.y)),
          pack_h2(__uint_as_float(vg.z), __uint_as_float(vg.w)),
          pack_h2(__uint_as_float(vh.z), __uint_as_float(vh.w)));
    }
  }
};

// ---- q5_0 / q4_1: the reference's default 131K configuration stores K as q5_0 and V as
// q4_1 (include/rdna4/kv.h:75-98); kv_load of kv.h:203-229 restated on fragments.
template <>
struct KLoad<RD_KV_Q5_0> {
  static constexpr float kUnscale = kQuantUnscale;
  // lane t owns blocks 2t and 2t+1 of the row: 44 bytes at 44t = eleven aligned words.
  // Block 2t is d | qh | 16 nibble bytes from byte 0, so its qh and nibble words straddle
  // two loaded words (realigned with PRMT); block 2t+1 starts at byte 22: d is the upper
  // half of word 5, qh is word 6 and the nibbles are words 7..10.
  __device__ static int dim(int t, int n, int e) {
    const int x = n >> 1;
    return (2 * t + (x >> 2)) * 32 + 4 * (x & 3) + (n & 1) + ((e & 1) ? 2 : 0) + ((e & 2) ? 16 : 0);
  }
  template <class F>
  __device__ static void run(uint32_t row_g, uint32_t row_h, int t, F &&mma) {
    uint32_t wg[11], wh[11];
#pragma unroll
    for (int i = 0; i < 11; ++i) {
      wg[i] = lds32(row_g + 44 * t + 4 * i);
      wh[i] = lds32(row_h + 44 * t + 4 * i);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const Q5Scale sg(b == 0 ? prmt(wg[0], wg[0], 0x1010u) : prmt(wg[5], wg[5], 0x3232u));
      const Q5Scale sh(b == 0 ? prmt(wh[0], wh[0], 0x1010u) : prmt(wh[5], wh[5], 0x3232u));
      const uint32_t qhg = b == 0 ? prmt(wg[0], wg[1], 0x5432u) : wg[6];
      const uint32_t qhh = b == 0 ? prmt(wh[0], wh[1], 0x5432u) : wh[6];
#pragma unroll
      for (int xx = 0; xx < 4; ++xx) {
        const int x = 4 * b + xx;
        const uint32_t xg = b == 0 ? prmt(wg[1 + xx], wg[2 + xx], 0x5432u) : wg[7 + xx];
        const uint32_t xh = b == 0 ? prmt(wh[1 + xx], wh[2 + xx], 0x5432u) : wh[7 + xx];
        uint32_t l0g, h0g, l1g, h1g, l0h, h0h, l1h, h1h;
        dq5(xg, (qhg >> (4 * xx)) & 0xFu, (qhg >> (16 + 4 * xx)) & 0xFu, sg, l0g, h0g, l1g, h1g);
        dq5(xh, (qhh >> (4 * xx)) & 0xFu, (qhh >> (16 + 4 * xx)) & 0xFu, sh, l0h, h0h, l1h, h1h);
        mma(2 * x, l0g, l0h, h0g, h0h);
        mma(2 * x + 1, l1g, l1h, h1g, h1h);
      }
    }
  }
};
template <>
struct KLoad<RD_KV_Q4_1> {
  static constexpr float kUnscale = kQuantUnscale;
  // lane t owns blocks t and t+4 of the row: five aligned words each ((d, m), then four
  // words of nibbles) at 20t and 20t + 80. (Blocks 2t and 2t+1 would put the four lanes
  // of a row 10 words apart: with the row pitch of 4 words mod 32 that is a 2-way bank
  // conflict on every load; 5 words apart is conflict-free.)
  __device__ static int dim(int t, int n, int e) {
    const int x = n >> 1;
    return (t + 4 * (x >> 2)) * 32 + 4 * (x & 3) + (n & 1) + ((e & 1) ? 2 : 0) + ((e & 2) ? 16 : 0);
  }
  template <class F>
  __device__ static void run(uint32_t row_g, uint32_t row_h, int t, F &&mma) {
#pragma unroll
    for (int b = 0; b < 2; ++b) {   // one block at a time: ten words live, not twenty
      uint32_t wg[5], wh[5];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        wg[i] = lds32(row_g + 20 * t + 80 * b + 4 * i);
        wh[i] = lds32(row_h + 20 * t + 80 * b + 4 * i);
      }
      const Q41Scale sg(prmt(wg[0], wg[0], 0x1010u), prmt(wg[0], wg[0], 0x3232u));
      const Q41Scale sh(prmt(wh[0], wh[0], 0x1010u), prmt(wh[0], wh[0], 0x3232u));
#pragma unroll
      for (int xx = 0; xx < 4; ++xx) {
        const int x = 4 * b + xx;
        uint32_t l0g, h0g, l1g, h1g, l0h, h0h, l1h, h1h;
        dq4(wg[1 + xx], sg, l0g, h0g, l1g, h1g);
        dq4(wh[1 + xx], sh, l0h, h0h, l1h, h1h);
        mma(2 * x, l0g, l0h, h0g, h0h);
        mma(2 * x + 1, l1g, l1h, h1g, h1h);
      }
    }
  }
};

// =============================== V loaders =======================================
// A fragment of V^T*P for M-tile m (0..15): rows g / g+8 = two true dims chosen by
// the loader (dim(g, m, r)), k-slots = keys (2t, 2t+1, 2t+8, 2t+9) of the group.
// kPairM says which two accumulator values of a lane are neighbours in memory (the
// epilogue stores them as one 8-byte word): true, dim(g, m + 1, r) = dim(g, m, r) + 1 for
// even m; false, dim(g, m, 1) = dim(g, m, 0) + 1. Either way the first dim is even.
// rows[j] is the shared address of the stored row of key j of those four. run()
// calls mma(m, a0, a1, a2, a3) for m = 0..15. Values come out multiplied by 1/kUnscale.
// run_part() does the M-tiles 4 * part .. 4 * part + 3 alone and numbers them 0..3.
template <int T>
struct VLoad;

template <>
struct VLoad<RD_KV_Q4_0> {
  static constexpr bool kPairM = true;
  static constexpr float kUnscale = kQuantUnscale;
  // lane g owns block g of each key: 18 bytes at 18g, read as 5 aligned words from
  // (18g & ~3); for odd g the block starts in the upper half of the first word.
  __device__ static int hidx(int s, int par) { return s <= 6 ? s + 1 - par : (par ? 7 : 0); }
  __device__ static int dim(int g, int m, int r) {
    return 32 * g + 2 * hidx(m >> 1, g & 1) + (m & 1) + (r ? 16 : 0);
  }
  template <class F>
  __device__ static void run(const uint32_t (&rows)[4], int g, F &&mma) {
    const uint32_t off = (18u * g) & ~3u;
    const bool par = g & 1;
    uint32_t w[4][5];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 5; ++i) w[j][i] = lds32(rows[j] + off + 4 * i);
    const uint32_t seld = par ? 0x7632u : 0x5410u;
    const uint32_t dab = prmt(w[0][0], w[1][0], seld);
    const uint32_t dcd = prmt(w[2][0], w[3][0], seld);
    const Q4Scale sab(dab), scd(dcd);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      uint32_t xab, xcd;
      if (s < 7) {
        const int i = 1 + (s >> 1);
        const uint32_t sel = (s & 1) ? 0x7632u : 0x5410u;
        xab = prmt(w[0][i], w[1][i], sel);
        xcd = prmt(w[2][i], w[3][i], sel);
      } else {
        xab = prmt(par ? w[0][4] : w[0][0], par ? w[1][4] : w[1][0], 0x7632u);
        xcd = prmt(par ? w[2][4] : w[2][0], par ? w[3][4] : w[3][0], 0x7632u);
      }
      uint32_t l0a, h0a, l1a, h1a, l0c, h0c, l1c, h1c;
      dq4(xab, sab, l0a, h0a, l1a, h1a);
      dq4(xcd, scd, l0c, h0c, l1c, h1c);
      mma(2 * s, l0a, h0a, l0c, h0c);
      mma(2 * s + 1, l1a, h1a, l1c, h1c);
    }
  }
  template <class F>
  __device__ static void run_part(const uint32_t (&rows)[4], int g, int part, F &&mma) {
    const uint32_t off = (18u * g) & ~3u;
    const bool par = g & 1;
    uint32_t w0[4], w1[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w0[j] = lds32(rows[j] + off);
      w1[j] = lds32(rows[j] + off + 4 + 4 * part);
    }
    const uint32_t seld = par ? 0x7632u : 0x5410u;
    const Q4Scale sab(prmt(w0[0], w0[1], seld)), scd(prmt(w0[2], w0[3], seld));
    const bool wrap = part == 3 && !par;   // slot 7 of an even block: the upper half of its first word
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const bool first = x == 1 && wrap;
      const uint32_t sel = x ? 0x7632u : 0x5410u;
      const uint32_t xab = prmt(first ? w0[0] : w1[0], first ? w0[1] : w1[1], sel);
      const uint32_t xcd = prmt(first ? w0[2] : w1[2], first ? w0[3] : w1[3], sel);
      uint32_t l0a, h0a, l1a, h1a, l0c, h0c, l1c, h1c;
      dq4(xab, sab, l0a, h0a, l1a, h1a);
      dq4(xcd, scd, l0c, h0c, l1c, h1c);
      mma(2 * x, l0a, h0a, l0c, h0c);
      mma(2 * x + 1, l1a, h1a, l1c, h1c);
    }
  }
};

template <>
struct VLoad<RD_KV_Q8_0> {
  static constexpr bool kPairM = false;
  static constexpr float kUnscale = kQuantUnscale;
  // lane g owns block g: 34 bytes at 34g, read as 9 aligned words from (34g & ~3).
  __device__ static int hidx(int s, int par) { return s <= 14 ? s + 1 - par : (par ? 15 : 0); }
  __device__ static int dim(int g, int m, int r) { return 32 * g + 2 * hidx(m, g & 1) + r; }
  template <class F>
  __device__ static void run(const uint32_t (&rows)[4], int g, F &&mma) {
    const uint32_t off = (34u * g) & ~3u;
    const bool par = g & 1;
    uint32_t w[4][9];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 9; ++i) w[j][i] = lds32(rows[j] + off + 4 * i);
    const uint32_t seld = par ? 0x7632u : 0x5410u;
    const uint32_t dab = prmt(w[0][0], w[1][0], seld);
    const uint32_t dcd = prmt(w[2][0], w[3][0], seld);
    const Q8Scale sab(dab), scd(dcd);
#pragma unroll
    for (int s = 0; s < 16; ++s) {
      uint32_t tab, tcd;  // bytes (a.b0, b.b0, a.b1, b.b1) of the 2-byte slot
      if (s < 15) {
        const int i = 1 + (s >> 1);
        const uint32_t sel = (s & 1) ? 0x7362u : 0x5140u;
        tab = prmt(w[0][i], w[1][i], sel);
        tcd = prmt(w[2][i], w[3][i], sel);
      } else {
        tab = prmt(par ? w[0][8] : w[0][0], par ? w[1][8] : w[1][0], 0x7362u);
        tcd = prmt(par ? w[2][8] : w[2][0], par ? w[3][8] : w[3][0], 0x7362u);
      }
      tab ^= 0x80808080u;
      tcd ^= 0x80808080u;
      uint32_t e0a, e1a, e0c, e1c;
      dq8(tab, sab, e0a, e1a);
      dq8(tcd, scd, e0c, e1c);
      mma(s, e0a, e1a, e0c, e1c);
    }
  }
  template <class F>
  __device__ static void run_part(const uint32_t (&rows)[4], int g, int part, F &&mma) {
    const uint32_t off = (34u * g) & ~3u;
    const bool par = g & 1;
    uint32_t w0[4], w1[4], w2[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w0[j] = lds32(rows[j] + off);
      w1[j] = lds32(rows[j] + off + 4 + 8 * part);
      w2[j] = lds32(rows[j] + off + 8 + 8 * part);
    }
    const uint32_t seld = par ? 0x7632u : 0x5410u;
    const Q8Scale sab(prmt(w0[0], w0[1], seld)), scd(prmt(w0[2], w0[3], seld));
    const bool wrap = part == 3 && !par;   // slot 15 of an even block: the upper half of its first word
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const bool first = x == 3 && wrap;
      const uint32_t sel = (x & 1) ? 0x7362u : 0x5140u;
      const uint32_t(&w)[4] = x < 2 ? w1 : w2;
      const uint32_t tab = prmt(first ? w0[0] : w[0], first ? w0[1] : w[1], sel) ^ 0x80808080u;
      const uint32_t tcd = prmt(first ? w0[2] : w[2], first ? w0[3] : w[3], sel) ^ 0x80808080u;
      uint32_t e0a, e1a, e0c, e1c;
      dq8(tab, sab, e0a, e1a);
      dq8(tcd, scd, e0c, e1c);
      mma(x, e0a, e1a, e0c, e1c);
    }
  }
};

template <>
struct VLoad<RD_KV_F16> {
  static constexpr bool kPairM = false;
  static constexpr float kUnscale = 1.0f;
  // lane g owns the 16-byte chunks g + 8*ci, ci = 0..3, of each key.
  __device__ static int dim(int g, int m, int r) { return 8 * (g + 8 * (m >> 2)) + 2 * (m & 3) + r; }
  template <class F>
  __device__ static void run(const uint32_t (&rows)[4], int g, F &&mma) {
#pragma unroll
    for (int ci = 0; ci < 4; ++ci) {
      const uint32_t o = 16 * (g + 8 * ci);
      const uint4 a = lds128(rows[0] + o), b = lds128(rows[1] + o);
      const uint4 c = lds128(rows[2] + o), d = lds128(rows[3] + o);
      mma(4 * ci + 0, prmt(a.x, b.x, 0x5410u), prmt(a.x, b.x, 0x7632u), prmt(c.x, d.x, 0x5410u),
          prmt(c.x, d.x, 0x7632u));
      mma(4 * ci + 1, prmt(a.y, b.y, 0x5410u), prmt(a.y, b.y, 0x7632u), prmt(c.y, d.y, 0x5410u),
          prmt(c.y, d.y, 0x7632u));
      mma(4 * ci + 2, prmt(a.z, b.z, 0x5410u), prmt(a.z, b.z, 0x7632u), prmt(c.z, d.z, 0x5410u),
          prmt(c.z, d.z, 0x7632u));
      mma(4 * ci + 3, prmt(a.w, b.w, 0x5410u), prmt(a.w, b.w, 0x7632u), prmt(c.w, d.w, 0x5410u),
          prmt(c.w, d.w, 0x7632u));
    }
  }
  template <class F>
  __device__ static void run_part(const uint32_t (&rows)[4], int g, int part, F &&mma) {
    const uint32_t o = 16 * (g + 8 * part);
    const uint4 a = lds128(rows[0] + o), b = lds128(rows[1] + o);
    const uint4 c = lds128(rows[2] + o), d = lds128(rows[3] + o);
    mma(0, prmt(a.x, b.x, 0x5410u), prmt(a.x, b.x, 0x7632u), prmt(c.x, d.x, 0x5410u), prmt(c.x, d.x, 0x7632u));
    mma(1, prmt(a.y, b.y, 0x5410u), prmt(a.y, b.y, 0x7632u), prmt(c.y, d.y, 0x5410u), prmt(c.y, d.y, 0x7632u));
    mma(2, prmt(a.z, b.z, 0x5410u), prmt(a.z, b.z, 0x7632u), prmt(c.z, d.z, 0x5410u), prmt(c.z, d.z, 0x7632u));
    mma(3, prmt(a.w, b.w, 0x5410u), prmt(a.w, b.w, 0x7632u), prmt(c.w, d.w, 0x5410u), prmt(c.w, d.w, 0x7632u));
  }
};

template <>
struct VLoad<RD_KV_F32> {
  static constexpr bool kPairM = false;
  static constexpr float kUnscale = 1.0f;
  // lane g owns the 16-byte chunks (4 dims) g + 8*ci, ci = 0..7.
  __device__ static int dim(int g, int m, int r) { return 4 * (g + 8 * (m >> 1)) + 2 * (m & 1) + r; }
  template <class F>
  __device__ static void run(const uint32_t (&rows)[4], int g, F &&mma) {
#pragma unroll
    for (int ci = 0; ci < 8; ++ci) {
      const uint32_t o = 16 * (g + 8 * ci);
      const uint4 a = lds128(rows[0] + o), b = lds128(rows[1] + o);
      const uint4 c = lds128(rows[2] + o), d = lds128(rows[3] + o);
#define RD_F(x) __uint_as_float(x)
      mma(2 * ci, pack_h2(RD_F(a.x), RD_F(b.x)), pack_h2(RD_F(a.y), RD_F(b.y)),
          pack_h2(RD_F(c.x), RD_F(d.x)), pack_h2(RD_F(c.y), RD_F(d.y)));
      mma(2 * ci + 1, pack_h2(RD_F(a.z), RD_F(b.z)), pack_h2(RD_F(a.w), RD_F(b.w)),
          pack_h2(RD_F(c.z), RD_F(d.z)), pack_h2(RD_F(c.w), RD_F(d.w)));
#undef RD_F
    }
  }
  template <class F>
  __device__ static void run_part(const uint32_t (&rows)[4], int g, int part, F &&mma) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const uint32_t o = 16 * (g + 8 * (2 * part + x));
      const uint4 a = lds128(rows[0] + o), b = lds128(rows[1] + o);
      const uint4 c = lds128(rows[2] + o), d = lds128(rows[3] + o);
#define RD_F(v) __uint_as_float(v)
      mma(2 * x, pack_h2(RD_F(a.x), RD_F(b.x)), pack_h2(RD_F(a.y), RD_F(b.y)), pack_h2(RD_F(c.x), RD_F(d.x)),
          pack_h2(RD_F(c.y), RD_F(d.y)));
      mma(2 * x + 1, pack_h2(RD_F(a.z), RD_F(b.z)), pack_h2(RD_F(a.w), RD_F(b.w)), pack_h2(RD_F(c.z), RD_F(d.z)),
          pack_h2(RD_F(c.w), RD_F(d.w)));
#undef RD_F
    }
  }
};

template <>
struct VLoad<RD_KV_Q5_0> {
  static constexpr bool kPairM = true;
  static constexpr float kUnscale = kQuantUnscale;
  // lane g owns block g of each key: 22 bytes at 22g, read as six aligned words from
  // (22g & ~3); for odd g the block starts in the upper half of the first word, which
  // shifts d, qh and the nibble words by two bytes (one PRMT selector per case).
  __device__ static int dim(int g, int m, int r) { return 32 * g + m + 16 * r; }
  template <class F>
  __device__ static void run(const uint32_t (&rows)[4], int g, F &&mma) {
    const uint32_t off = (22u * g) & ~3u;
    const bool par = g & 1;
    const uint32_t sel = par ? 0x7654u : 0x5432u;   // odd g: the next word is already aligned
    uint32_t dd[4], qh[4], qs[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t w[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) w[i] = lds32(rows[j] + off + 4 * i);
      dd[j] = prmt(w[0], w[0], par ? 0x3232u : 0x1010u);
      qh[j] = prmt(w[0], w[1], sel);
#pragma unroll
      for (int x = 0; x < 4; ++x) qs[j][x] = prmt(w[1 + x], w[2 + x], sel);
    }
    const Q5Scale sab(prmt(dd[0], dd[1], 0x5410u)), scd(prmt(dd[2], dd[3], 0x5410u));
    // fifth bits of element pairs, two keys side by side: nibble (s & ~1) * 2 of pe (even
    // slots s) / po (odd slots) holds (key0 bits 2s, 2s+1 | key1 bits 2s, 2s+1)
    const uint32_t pe_ab = (qh[0] & 0x33333333u) | ((qh[1] & 0x33333333u) << 2);
    const uint32_t po_ab = ((qh[0] >> 2) & 0x33333333u) | (qh[1] & 0xCCCCCCCCu);
    const uint32_t pe_cd = (qh[2] & 0x33333333u) | ((qh[3] & 0x33333333u) << 2);
    const uint32_t po_cd = ((qh[2] >> 2) & 0x33333333u) | (qh[3] & 0xCCCCCCCCu);
#pragma unroll
    for (int s = 0; s < 8; ++s) {   // bytes 2s, 2s+1 of the nibbles: elements 2s, 2s+1 (+16)
      const uint32_t psel = (s & 1) ? 0x7632u : 0x5410u;
      const uint32_t xab = prmt(qs[0][s >> 1], qs[1][s >> 1], psel);
      const uint32_t xcd = prmt(qs[2][s >> 1], qs[3][s >> 1], psel);
      const int sh = 4 * (s >> 1);
      const uint32_t bab = (s & 1) ? po_ab : pe_ab, bcd = (s & 1) ? po_cd : pe_cd;
      uint32_t l0a, h0a, l1a, h1a, l0c, h0c, l1c, h1c;
      dq5(xab, (bab >> sh) & 0xFu, (bab >> (16 + sh)) & 0xFu, sab, l0a, h0a, l1a, h1a);
      dq5(xcd, (bcd >> sh) & 0xFu, (bcd >> (16 + sh)) & 0xFu, scd, l0c, h0c, l1c, h1c);
      mma(2 * s, l0a, h0a, l0c, h0c);
      mma(2 * s + 1, l1a, h1a, l1c, h1c);
    }
  }
  template <class F>
  __device__ static void run_part(const uint32_t (&rows)[4], int g, int part, F &&mma) {
    const uint32_t off = (22u * g) & ~3u;
    const bool par = g & 1;
    const uint32_t sel = par ? 0x7654u : 0x5432u;   // odd g: the next word is already aligned
    uint32_t dd[4], qh[4], qs[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t w0 = lds32(rows[j] + off), w1 = lds32(rows[j] + off + 4);
      const uint32_t a = lds32(rows[j] + off + 4 + 4 * part), b = lds32(rows[j] + off + 8 + 4 * part);
      dd[j] = prmt(w0, w0, par ? 0x3232u : 0x1010u);
      qh[j] = prmt(w0, w1, sel);
      qs[j] = prmt(a, b, sel);
    }
    const Q5Scale sab(prmt(dd[0], dd[1], 0x5410u)), scd(prmt(dd[2], dd[3], 0x5410u));
    const int sh = 4 * part;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const uint32_t psel = x ? 0x7632u : 0x5410u;
      const uint32_t xab = prmt(qs[0], qs[1], psel), xcd = prmt(qs[2], qs[3], psel);
      // fifth bits of two elements, two keys side by side (see run)
      const uint32_t bab = x ? ((qh[0] >> 2) & 0x33333333u) | (qh[1] & 0xCCCCCCCCu)
                             : (qh[0] & 0x33333333u) | ((qh[1] & 0x33333333u) << 2);
      const uint32_t bcd = x ? ((qh[2] >> 2) & 0x33333333u) | (qh[3] & 0xCCCCCCCCu)
                             : (qh[2] & 0x33333333u) | ((qh[3] & 0x33333333u) << 2);
      uint32_t l0a, h0a, l1a, h1a, l0c, h0c, l1c, h1c;
      dq5(xab, (bab >> sh) & 0xFu, (bab >> (16 + sh)) & 0xFu, sab, l0a, h0a, l1a, h1a);
      dq5(xcd, (bcd >> sh) & 0xFu, (bcd >> (16 + sh)) & 0xFu, scd, l0c, h0c, l1c, h1c);
      mma(2 * x, l0a, h0a, l0c, h0c);
      mma(2 * x + 1, l1a, h1a, l1c, h1c);
    }
  }
};
template <>
struct VLoad<RD_KV_Q4_1> {
  static constexpr bool kPairM = true;
  static constexpr float kUnscale = kQuantUnscale;
  // lane g owns block g of each key: 20 bytes at 20g = five aligned words.
  __device__ static int dim(int g, int m, int r) { return 32 * g + m + 16 * r; }
  template <class F>
  __device__ static void run(const uint32_t (&rows)[4], int g, F &&mma) {
    uint32_t w[4][5];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 5; ++i) w[j][i] = lds32(rows[j] + 20u * g + 4 * i);
    // half2 across two keys: (key a, key b) and (key c, key d), each with its own (d, m)
    const Q41Scale sab(prmt(w[0][0], w[1][0], 0x5410u), prmt(w[0][0], w[1][0], 0x7632u));
    const Q41Scale scd(prmt(w[2][0], w[3][0], 0x5410u), prmt(w[2][0], w[3][0], 0x7632u));
#pragma unroll
    for (int s = 0; s < 8; ++s) {   // bytes 2s, 2s+1 of the nibbles: elements 2s, 2s+1 (+16)
      const int i = 1 + (s >> 1);
      const uint32_t sel = (s & 1) ? 0x7632u : 0x5410u;
      const uint32_t xab = prmt(w[0][i], w[1][i], sel);
      const uint32_t xcd = prmt(w[2][i], w[3][i], sel);
      uint32_t l0a, h0a, l1a, h1a, l0c, h0c, l1c, h1c;
      dq4(xab, sab, l0a, h0a, l1a, h1a);
      dq4(xcd, scd, l0c, h0c, l1c, h1c);
      mma(2 * s, l0a, h0a, l0c, h0c);
      mma(2 * s + 1, l1a, h1a, l1c, h1c);
    }
  }
  template <class F>
  __device__ static void run_part(const uint32_t (&rows)[4], int g, int part, F &&mma) {
    uint32_t w0[4], w1[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w0[j] = lds32(rows[j] + 20u * g);
      w1[j] = lds32(rows[j] + 20u * g + 4 + 4 * part);
    }
    const Q41Scale sab(prmt(w0[0], w0[1], 0x5410u), prmt(w0[0], w0[1], 0x7632u));
    const Q41Scale scd(prmt(w0[2], w0[3], 0x5410u), prmt(w0[2], w0[3], 0x7632u));
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const uint32_t sel = x ? 0x7632u : 0x5410u;
      uint32_t l0a, h0a, l1a, h1a, l0c, h0c, l1c, h1c;
      dq4(prmt(w1[0], w1[1], sel), sab, l0a, h0a, l1a, h1a);
      dq4(prmt(w1[2], w1[3], sel), scd, l0c, h0c, l1c, h1c);
      mma(2 * x, l0a, h0a, l0c, h0c);
      mma(2 * x + 1, l1a, h1a, l1c, h1c);
    }
  }
};

}  // namespace rd
