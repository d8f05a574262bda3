// Dequantisation of 32 values of one weight row from a packed super-block in shared memory, for the tensor-core kernels: as
// packed bf16 pairs in one piece (rounded once) or in two that add up to the value within 2^-18.
//
// The code is written to be SMALL: which 32 values (j = 0..7 of a super-block's 256) is a run-time argument and the callers'
// loops stay rolled (one_piece: one 64-value group).  Sixteen warps that run straight through unrolled code for every j and nibble half starve on
// instruction fetch: of 10.5 warps resident per scheduler 3.2 waited for instructions, and a K step of the two-piece kernel
// took 0.85 us whatever the number of producer warps.
#pragma once

#include "tc.cuh"

namespace ub {

enum { kQ4K = 0, kQ8 = 1, kQ6K = 2, kQ5K = 3, kQ40 = 4 };

// bytes of 256 values in memory / per row of a slot of a packed ring / of a slot (Q6_K: 224 of the 240 bytes are read, with
// rows 224 bytes apart a quarter of the banks would serve all rows; eight more rows per slot)
constexpr uint32_t row_sb_bytes(int f) { return f == kQ8 ? 272 : f == kQ6K ? 210 : f == kQ5K ? 176 : 144; }
constexpr uint32_t slot_pitch(int f) { return f == kQ6K ? 240 : row_sb_bytes(f); }
constexpr uint32_t slot_bytes(int f) { return (f == kQ6K ? 136 : 128) * slot_pitch(f); }

// Two bytes A and B of a word -> packed bf16 (s * byte + c).  A byte n with nothing above it is the bf16 n * 2^-133, below 128
// a subnormal, from there on the first normal binade, which has the same spacing: no bias to subtract.  s carries 2^133.
template <int SEL>
__device__ __forceinline__ uint32_t deq_pair(uint32_t w4, __nv_bfloat162 s, __nv_bfloat162 c) {
  const uint32_t n = __byte_perm(w4, 0u, SEL);
  return bf162_bits(__hfma2(*reinterpret_cast<const __nv_bfloat162*>(&n), s, c));
}

// The same with s of any size: the byte times 2^-6 first (exact), s carries 2^6.
template <int SEL>
__device__ __forceinline__ uint32_t deq_pair_wide(uint32_t w4, __nv_bfloat162 s, __nv_bfloat162 c) {
  const uint32_t n = __byte_perm(w4, 0u, SEL), big = 0x7F007F00u;  // 2^127
  const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&n), *reinterpret_cast<const __nv_bfloat162*>(&big));
  return bf162_bits(__hfma2(v, s, c));
}

// Two signed bytes A and B of a word (given with their sign bits flipped: q + 128) -> packed bf16 (d * q): q 2^-6 from the bf16
// n * 2^-133 in one exact step (2^127 n 2^-133 - 2), then d in two pieces, which carry 2^6: fma(q, dh, q dl) is d q rounded once.
template <int SEL>
__device__ __forceinline__ uint32_t deq8_pair(uint32_t u4, __nv_bfloat162 dh, __nv_bfloat162 dl) {
  const uint32_t n = __byte_perm(u4, 0u, SEL), big = 0x7F007F00u, two = 0xC000C000u;
  const __nv_bfloat162 q = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&n), *reinterpret_cast<const __nv_bfloat162*>(&big),
                                   *reinterpret_cast<const __nv_bfloat162*>(&two));
  return bf162_bits(__hfma2(q, dh, __hmul2(q, dl)));
}

// Two floats -> two packed bf16 pairs that add up to them (a in the lower half): rounded and remainder, or ...
__device__ __forceinline__ void split_rn(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = bf162_bits(__floats2bfloat162_rn(a, b));
  lo = bf162_bits(__floats2bfloat162_rn(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xFFFF0000u)));
}
// ... upper halves and remainder (no overflow near the largest float)
__device__ __forceinline__ void split_cut(float a, float b, uint32_t& hi, uint32_t& lo) {
  const uint32_t ua = __float_as_uint(a), ub_ = __float_as_uint(b);
  hi = __byte_perm(ua, ub_, 0x7632);
  lo = bf162_bits(__floats2bfloat162_rn(a - __uint_as_float(ua & 0xFFFF0000u), b - __uint_as_float(ub_ & 0xFFFF0000u)));
}

// Four unsigned bytes q < 128 of a word -> s * q - m in two pieces, c = 128 s + m.  0x43 in the top byte and q below it
// is the float 128 + q.
__device__ __forceinline__ void deq4(uint32_t w4, float s, float c, uint32_t* hi, uint32_t* lo) {
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = fmaf(s, __uint_as_float(__byte_perm(w4, 0x43000000u, 0x7044u | (i << 8))), -c);
  split_rn(v[0], v[1], hi[0], lo[0]);
  split_rn(v[2], v[3], hi[1], lo[1]);
}
// Four signed bytes (given with their sign bits flipped) -> s * q; 0x4B in the top byte and u in the lowest is 2^23 + u.
__device__ __forceinline__ void deq4_signed(uint32_t u4, float s, uint32_t* hi, uint32_t* lo) {
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = s * (__uint_as_float(__byte_perm(u4, 0x4B000000u, 0x7440u | i)) - 8388736.f);
  split_rn(v[0], v[1], hi[0], lo[0]);
  split_rn(v[2], v[3], hi[1], lo[1]);
}

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}


__device__ __forceinline__ void lds128(uint32_t a, uint32_t* v) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a));
}
__device__ __forceinline__ int lds_s8(uint32_t a) {
  int v;
  asm volatile("ld.shared.s8 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}

// What the two forms cost, B200, 16 warps per SM, cycles for 256 values of 128 rows with the tcgen05.st: Q4_K one piece 636
// (884 while the nibbles were biased by 128 and the bias subtracted: byte permutes, logic and 16-bit arithmetic all issue at half
// rate, ten instructions per eight values now take 12 cycles of the one pipe and 8 of the other instead of 14 and 16), two
// pieces 2100.  It is the largest part of a launch of few tokens: 16 tokens through 28672x4096 26.4 -> 23.9 us, Q8_0 45 tokens
// 14336x4096 24.8 -> 21.8 us.
//
// One piece of Q4_K: low nibbles as q 2^-133, high ones as 16 q 2^-133, and a scale that carries the rest, finite in bf16 while a
// super-block's d is below this (63 * 2^-11 * 2^133 < 2^128; trained weights have d of 1e-5 to 4e-4).  Where a row of the warp has a
// larger one, the nibbles are multiplied by 2^127 first, exactly: two instructions more per four values, up to 10 % of a launch.
// Both give bf16(s q - m), s and m rounded to bf16, and accumulators of ordinary size: with a factor on all weights instead, taken back
// from the sums, products of activations below 2^-92 would be subnormal.  The choice costs 0 to 1.5 % (expert layers of a few hundred
// rows per expert most), and 3 % when made anew for each nibble half and from the f32 scale.  Low nibbles moved up by four bits
// would do until 2^-7, for another 0.7 %.
constexpr uint32_t kOnePieceMaxD = 0x1000;  // 2^-11 in f16

template <int FMT>
struct RowBlock {
  uint32_t base;  // shared-memory address of the row's block: 16-byte aligned, Q6_K: 2-byte aligned
  uint32_t scw[2], mnw[2], fifth[8];
  float d, dmin;
  bool wide;  // Q4_K: of any row of the warp

  __device__ __forceinline__ void open(uint32_t at) {
    base = at;
    if constexpr (FMT == kQ4K || FMT == kQ5K) {
      uint32_t h[4];
      lds128(base, h);
      d = half_bits_to_f32(h[0]), dmin = half_bits_to_f32(h[0] >> 16);
      q4k_unpack_scales(h[1], h[2], h[3], scw[0], scw[1], mnw[0], mnw[1]);
      if constexpr (FMT == kQ4K) wide = __any_sync(0xFFFFFFFFu, (h[0] & 0x7FFFu) >= kOnePieceMaxD);
      if constexpr (FMT == kQ5K) lds128(base + 16, fifth), lds128(base + 32, fifth + 4);  // of all eight sub-blocks
    }
    if constexpr (FMT == kQ6K) d = half_bits_to_f32(lds32((base + 208) & ~3u) >> ((base & 2) * 8));
  }
  // scale and min of sub-block j (Q4_K, Q5_K)
  __device__ __forceinline__ void pair(int j, float& s, float& m) const {
    // 0x4B in the top byte and the 6-bit number in the lowest is 2^23 + number: no conversion instruction
    s = d * (__uint_as_float((__byte_perm(scw[0], scw[1], j) & 0xFFu) | 0x4B000000u) - 8388608.f);
    m = dmin * (__uint_as_float((__byte_perm(mnw[0], mnw[1], j) & 0xFFu) | 0x4B000000u) - 8388608.f);
  }
  // N words from byte `off` of the shared-memory words around it; off is a multiple of 2
  template <int N>
  static __device__ __forceinline__ void words(uint32_t at, uint32_t (&v)[N]) {
    const uint32_t p = at & ~3u, sh = (at & 2) * 8;
    uint32_t prev = lds32(p);
#pragma unroll
    for (int i = 0; i < N; i++) {
      const uint32_t next = lds32(p + 4 * i + 4);
      v[i] = __funnelshift_r(prev, next, sh);
      prev = next;
    }
  }

  // values 64 G .. 64 G + 63 in order, rounded to bf16 once (Q4_K and Q8_0).  A whole 64-value group per thread: the words
  // of a Q4_K group serve both nibble halves, and which half is a compile-time shift.
  __device__ __forceinline__ void one_piece(int G, uint32_t (&ot)[32]) const {
    static_assert(FMT == kQ4K || FMT == kQ8, "formats with a one-piece producer");
    if constexpr (FMT == kQ4K) {
      uint32_t q[8];
      lds128(base + 16 + 32 * G, q), lds128(base + 32 + 32 * G, q + 4);
      if (__builtin_expect(!wide, 1)) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          float s, m;
          pair(2 * G + h, s, m);
          const __nv_bfloat162 dsc = __float2bfloat162_rn(s * (h ? 0x1p65f : 0x1p69f) * 0x1p64f), ndm = __float2bfloat162_rn(-m);
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const uint32_t v = q[i] & (h ? 0xF0F0F0F0u : 0x0F0F0F0Fu);
            ot[16 * h + 2 * i] = deq_pair<0x4140>(v, dsc, ndm);
            ot[16 * h + 2 * i + 1] = deq_pair<0x4342>(v, dsc, ndm);
          }
        }
      } else {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          float s, m;
          pair(2 * G + h, s, m);
          const __nv_bfloat162 dsc = __float2bfloat162_rn(s * (h ? 4.f : 64.f)), ndm = __float2bfloat162_rn(-m);
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const uint32_t v = q[i] & (h ? 0xF0F0F0F0u : 0x0F0F0F0Fu);
            ot[16 * h + 2 * i] = deq_pair_wide<0x4140>(v, dsc, ndm);
            ot[16 * h + 2 * i + 1] = deq_pair_wide<0x4342>(v, dsc, ndm);
          }
        }
      }
    } else {
      // two blocks of 34 bytes at 68 G; the first one's words straddle two loaded words
      const uint32_t at = base + 68 * G;
      uint32_t prev = lds32(at);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const float df = 64.f * half_bits_to_f32(h ? prev >> 16 : prev);
        const __nv_bfloat16 dh1 = __float2bfloat16_rn(df);
        const __nv_bfloat162 dh = __bfloat162bfloat162(dh1), dl = __float2bfloat162_rn(df - __bfloat162float(dh1));
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const uint32_t next = lds32(at + 32 * h + 4 * i + 4);
          const uint32_t u = (h ? next : __funnelshift_r(prev, next, 16)) ^ 0x80808080u;
          prev = next;
          ot[16 * h + 2 * i] = deq8_pair<0x4140>(u, dh, dl);
          ot[16 * h + 2 * i + 1] = deq8_pair<0x4342>(u, dh, dl);
        }
      }
    }
  }

  // values 32 j .. 32 j + 31 in order, in two pieces
  __device__ __forceinline__ void two_pieces(int j, uint32_t (&hi)[16], uint32_t (&lo)[16]) const {
    if constexpr (FMT == kQ4K || FMT == kQ5K) {
      float s, m;
      pair(j, s, m);
      const float c = fmaf(s, 128.f, m);
      const uint32_t at = base + (FMT == kQ5K ? 48 : 16) + 32 * (j >> 1);
      uint32_t q[8];
      lds128(at, q), lds128(at + 16, q + 4);
      const int sh = 4 * (j & 1);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        uint32_t v = (q[i] >> sh) & 0x0F0F0F0Fu;
        if (FMT == kQ5K) v += ((fifth[i] >> j) & 0x01010101u) * 16u;
        deq4(v, s, c, hi + 2 * i, lo + 2 * i);
      }
    } else if constexpr (FMT == kQ40) {
      const uint32_t at = base + 18 * j;
      uint32_t q[4];
      words(at + 2, q);
      const float s = half_bits_to_f32(lds32(at & ~3u) >> ((at & 2) * 8)), c = 136.f * s;
#pragma unroll
      for (int i = 0; i < 4; i++) {  // bytes 0-15: values 0-15 in the low nibbles, 16-31 in the high ones
        deq4(q[i] & 0x0F0F0F0Fu, s, c, hi + 2 * i, lo + 2 * i);
        deq4((q[i] >> 4) & 0x0F0F0F0Fu, s, c, hi + 8 + 2 * i, lo + 8 + 2 * i);
      }
    } else if constexpr (FMT == kQ6K) {
      // nibbles in ql bytes 64 (j / 4) + 32 (j % 2) .., upper halves for j % 4 >= 2; top bits at 2 (j % 4) of the qh bytes
      // 32 (j / 4) ..; one int8 scale per 16 values
      uint32_t ql[8], qh[8];
      words(base + 64 * (j >> 2) + 32 * (j & 1), ql);
      words(base + 128 + 32 * (j >> 2), qh);
      const int sn = 2 * (j & 2), st = 2 * (j & 3);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const float s = d * static_cast<float>(lds_s8(base + 192 + 2 * j + u)), c = 160.f * s;
#pragma unroll
        for (int i = 4 * u; i < 4 * u + 4; i++)
          deq4(((ql[i] >> sn) & 0x0F0F0F0Fu) + ((qh[i] >> st) & 0x03030303u) * 16u, s, c, hi + 2 * i, lo + 2 * i);
      }
    } else {
      const uint32_t at = base + 34 * j;
      uint32_t w[8];
      words(at + 2, w);
      const float s = half_bits_to_f32(lds32(at & ~3u) >> ((at & 2) * 8));
#pragma unroll
      for (int i = 0; i < 8; i++) deq4_signed(w[i] ^ 0x80808080u, s, hi + 2 * i, lo + 2 * i);
    }
  }
};

}  // namespace ub
