// Matmul of a few tokens on the tensor cores (tcgen05 / TMEM) with the weights' integers as they are.
//
//   y[M,N] (f32 / bf16 / f16) = x[M,K] (bf16 or f32) . dequant(Wq)^T,   f32 accumulation
//
// The reference declares these block formats (kernels/quant.cpp:64-178) and multiplies dequantised copies
// (kernels/matmul.cpp:1143-1184).  Here a weight is never dequantised.  Within a group of 32 values (Q6_K: 16) a weight is
// s * u + b, u a small integer, s and b the group's own: the sum over the group is s * sum(u x) + b * sum(x).  The integers go
// to the tensor cores as bf16 (exact), every group has an accumulator of its own, and s and b are applied in f32 to the
// groups' sums.  Activations are exact too: bf16 ones come as they are, f32 ones in three bf16 pieces (24 bits), so results
// carry f32 rounding only: 0.5e-7 to 1.2e-7 of a result as a 2-norm, 256 to 14336 values (CUDA-core kernels 0.6e-7 to 3.9e-7,
// integer kernels with 15-bit activations 2.8e-5, two-piece weights 2e-6 to 2.6e-5).  An infinite activation gives what the plain
// sum gives (sum_of_infinities), a NaN gives NaN.
//
// u is centred (Q4_K and Q4_0 q - 8, Q5_K q - 16, Q6_K q - 32, Q8_0 signed): small sums lose least when a result is small, and
// Q4_0, Q6_K and Q8_0 have no second term.  The tensor cores get 2^-8 u, so that sums of large activations do not
// overflow before the scale is applied; 2^8 goes into the scale.
//
// A CTA takes 128 weight rows x 16 tokens, K in stages of 128 values (Q6_K: 64), two CTAs per SM:
//   warps 0-7     integers: a thread reads its row's packed super-block from shared memory and writes bf16 pairs into tensor
//                 memory (tcgen05.st); each set of four warps has a stage of its own
//   warps 8-11    sums: a thread takes its row's group sums from tensor memory (tcgen05.ld), scale and offset of the group
//                 from the packed super-block, the groups' activation sums from shared memory, and keeps the tokens in registers
//   warps 12, 13  one lane each issues tcgen05.mma (A from tensor memory, B from shared memory) and tcgen05.commit for one of
//                 the two stages
//   warp 14       copies of packed weights, one super-block column (256 values of 128 rows) each, and of bf16 token tiles
//   warp 15       (bf16 activations, formats with b) sums of the activations of every group: mma.sync with ones
//   warps 15, 16  (f32 activations) the token tile's three pieces and the groups' sums
//
// What bounds it: the sums' chain, 2100 cycles per super-block and CTA with four tokens (two barriers 500, scales and offsets
// 600, two reads of tensor memory 700), two CTAs per SM, where the copies of a super-block take 790 cycles of an SM's share of
// the memory and the integers 570.  The variants of sixteen tokens also spill registers (60 to 206 bytes a thread).
// Measured on B200, us, before / this kernel: Q4_K four tokens 4096x14336 30.6 / 15.4, Q8_0 four 6144x5120 76 / 12.2, Q5_K ten
// tokens, f32 results, 2688x7680 284 / 15.1.
//
// K split.  A tile may belong to a cluster of up to eight CTAs, each with a part of K.  Every CTA owns some of the 128 rows
// and gets the others' partial sums of them (st.async, counted in bytes on a barrier of the owner); it adds them in a fixed
// order: deterministic.
//
// Every wait is bounded; on expiry the CTA records UB_ERR_TIMEOUT, all roles leave and TMEM is freed.
#include <string.h>

#include "rowblock.cuh"

namespace ub {
void* tensor_map_encoder();
bool q4_0_staged_takes(int M, int K);
bool q5k_staged_takes(int M, int K);
bool q6k_staged_takes(int M, int K);
bool q4k_imma_takes(int M, int K);
bool q8_0_imma_takes(int M, int K);
int two_piece_split(int tiles, int nsb);
}

namespace {

using namespace ub;

constexpr int kTok = 16;       // tokens of a tile: N of the MMAs
constexpr int kMaxX = 3, kMaxW = 4;
constexpr int kStages = 2;     // stages in tensor memory
constexpr uint32_t kTmemCols = 256;

constexpr int x_vals(bool xf) { return xf ? 128 : 256; }  // values of an activation slot
constexpr int stage_vals(int f) { return f == kQ6K ? 64 : 128; }
constexpr bool has_offset(int f) { return f == kQ4K || f == kQ5K; }
// f32: two, so that each of the MMA warps and of the converting warps keeps to one (a wait by parity must not skip a round)
constexpr int x_slots(bool xf) { return xf ? 2 : 3; }
constexpr uint32_t x_bytes(bool xf) { return kTok * x_vals(xf) * 2 * (xf ? 3 : 1); }
constexpr int w_slots(int f) { return f == kQ4K || f == kQ40 ? 4 : f == kQ5K ? 3 : 2; }
constexpr int threads_of(bool xf) { return (xf ? 17 : 16) * 32; }
constexpr uint32_t kRecvBytes = (128 + 8) * kTok * 4;
// Rounding.  A chain of n additions rounds n / 2 times as much as one.  Without an offset a stage of four groups is summed by itself,
// then the stages of a super-block, then super-blocks.  Q6_K has twice the groups, and what an addition of a super-block
// rounds off is summed beside it, in shared memory (in registers it would spill more).  Q6_K takes longer for it: four tokens 1 %, eight
// 3 to 5 %, sixteen 2 to 13 % (28672x5120 65.7 -> 70.7 us).  Error of f32 results as a part of the CUDA-core kernels', bf16
// activations: Q6_K 1200 rows of 1536 values 0.98 (1.20 in one chain per super-block), 24000 rows of 4352 values 0.75 (1.14 without
// the rest), Q8_0 1024 values 0.97 (1.04 in one chain).
constexpr bool keeps_stages(int f) { return f == kQ6K || f == kQ8; }
constexpr bool keeps_rest(int f) { return f == kQ6K; }
constexpr uint32_t rest_bytes(int f) { return keeps_rest(f) ? 128 * kTok * 4 : 0; }
constexpr size_t smem_of(int f, bool xf) {
  return static_cast<size_t>(x_slots(xf)) * (x_bytes(xf) + x_vals(xf) * 2) + static_cast<size_t>(w_slots(f)) * slot_bytes(f) +
         kRecvBytes + rest_bytes(f) + 1024;
}

struct SharedU {
  unsigned long long wfull[kMaxW], wempty[kMaxW], xfull[kMaxX], xempty[kMaxX], sfull[kMaxX];
  unsigned long long afull[kStages], done[kStages], dempty[kStages];
  unsigned long long pfull;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void st_async16(uint32_t peer_addr, const float* v, uint32_t peer_bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(peer_addr),
      "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
      "r"(peer_bar)
      : "memory");
}

__device__ __forceinline__ void store_one(void* y, size_t at, int dtype, float v) {
  if (dtype == UB_DTYPE_F32)
    static_cast<float*>(y)[at] = v;
  else if (dtype == UB_DTYPE_BF16)
    static_cast<__nv_bfloat16*>(y)[at] = __float2bfloat16_rn(v);
  else
    static_cast<__half*>(y)[at] = __float2half_rn(v);
}

__device__ __forceinline__ float load_one(const void* y, size_t at, int dtype) {
  if (dtype == UB_DTYPE_F32) return static_cast<const float*>(y)[at];
  if (dtype == UB_DTYPE_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(y)[at]);
  return __half2float(static_cast<const __half*>(y)[at]);
}
// of the first n
template <int N>
__device__ __forceinline__ bool all_finite(const float (&v)[N], int n) {
  float zero = 0.f;
#pragma unroll
  for (int i = 0; i < N; i++) zero = fmaf(i < n ? v[i] : 0.f, 0.f, zero);
  return zero == 0.f;
}

// Several barriers at once: one look at each costs some 200 cycles however long ago the phase ended, and the looks overlap.
__device__ __forceinline__ bool wait2(uint32_t a, uint32_t pa, uint32_t b, uint32_t pb, volatile int* abort_flag) {
  const bool ra = tc_mbar_test(a, pa), rb = tc_mbar_test(b, pb);
  return (ra || tc_wait(a, pa, abort_flag)) && (rb || tc_wait(b, pb, abort_flag));
}
__device__ __forceinline__ bool wait3(uint32_t a, uint32_t pa, uint32_t b, uint32_t pb, uint32_t c, uint32_t pc,
                                      volatile int* abort_flag) {
  const bool ra = tc_mbar_test(a, pa), rb = tc_mbar_test(b, pb), rc = tc_mbar_test(c, pc);
  return (ra || tc_wait(a, pa, abort_flag)) && (rb || tc_wait(b, pb, abort_flag)) && (rc || tc_wait(c, pc, abort_flag));
}

// N consecutive accumulator columns (N = 4, 8, 16)
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[N]) {
  uint32_t r[N];
  if constexpr (N == 4)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
  else if constexpr (N == 8)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
  else
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
  for (int i = 0; i < N; i++) v[i] = __uint_as_float(r[i]);
}

// (a0, a1) += (b0, b1) * (c, c), both products in one instruction
__device__ __forceinline__ void fma2(float& a0, float& a1, float b0, float b1, float c) {
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tmov.b64 c, {%4, %4};\n\t"
      "fma.rn.f32x2 a, b, c, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "f"(b0), "f"(b1), "f"(c));
}
__device__ __forceinline__ void mul2(float& a0, float& a1, float b0, float b1, float c) {
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 b, {%2, %3};\n\tmov.b64 c, {%4, %4};\n\t"
      "mul.rn.f32x2 a, b, c;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "=f"(a0), "=f"(a1)
      : "f"(b0), "f"(b1), "f"(c));
}

// Integers of 64 consecutive values of a row as bf16 pairs of 2^-8 u.  A byte n with nothing above it is the bf16 n * 2^-133
// (rowblock.cuh): one exact multiply-add scales it and takes the centre off.
template <int FMT>
struct UnitRow {
  uint32_t base;

  __device__ __forceinline__ void open(uint32_t at) { base = at; }
  // four bytes n of a word -> 2^-8 (n / 2^SHIFT - CENTRE)
  template <int CENTRE, int SHIFT>
  static __device__ __forceinline__ void four(uint32_t w4, uint32_t& a, uint32_t& b) {
    constexpr uint32_t scale = (252u - SHIFT) << 7;  // 2^(125 - SHIFT)
    constexpr uint32_t c = CENTRE == 8 ? 0xBD00u : CENTRE == 16 ? 0xBD80u : CENTRE == 32 ? 0xBE00u : 0xBF00u;  // 128: -0.5
    static_assert(CENTRE == 8 || CENTRE == 16 || CENTRE == 32 || CENTRE == 128, "centre");
    const uint32_t s2 = scale | scale << 16, c2 = c | c << 16;
    const uint32_t pa = __byte_perm(w4, 0u, 0x4140), pb = __byte_perm(w4, 0u, 0x4342);
    const __nv_bfloat162 sv = *reinterpret_cast<const __nv_bfloat162*>(&s2), cv = *reinterpret_cast<const __nv_bfloat162*>(&c2);
    a = bf162_bits(__hfma2(*reinterpret_cast<const __nv_bfloat162*>(&pa), sv, cv));
    b = bf162_bits(__hfma2(*reinterpret_cast<const __nv_bfloat162*>(&pb), sv, cv));
  }

  __device__ __forceinline__ void group64(int G, uint32_t (&ot)[32]) const {
    if constexpr (FMT == kQ4K) {
      uint32_t q[8];
      lds128(base + 16 + 32 * G, q), lds128(base + 32 + 32 * G, q + 4);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        four<8, 0>(q[i] & 0x0F0F0F0Fu, ot[2 * i], ot[2 * i + 1]);
        four<8, 4>(q[i] & 0xF0F0F0F0u, ot[16 + 2 * i], ot[16 + 2 * i + 1]);
      }
    } else if constexpr (FMT == kQ5K) {
      uint32_t q[8], fifth[8];
      lds128(base + 48 + 32 * G, q), lds128(base + 64 + 32 * G, q + 4);
      lds128(base + 16, fifth), lds128(base + 32, fifth + 4);
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < 8; i++)
          four<16, 0>(((h ? q[i] >> 4 : q[i]) & 0x0F0F0F0Fu) | ((fifth[i] >> (2 * G + h)) & 0x01010101u) * 16u,
                      ot[16 * h + 2 * i], ot[16 * h + 2 * i + 1]);
    } else if constexpr (FMT == kQ40) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint32_t q[4];
        RowBlock<FMT>::words(base + 36 * G + 18 * h + 2, q);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          four<8, 0>(q[i] & 0x0F0F0F0Fu, ot[16 * h + 2 * i], ot[16 * h + 2 * i + 1]);
          four<8, 4>(q[i] & 0xF0F0F0F0u, ot[16 * h + 8 + 2 * i], ot[16 * h + 8 + 2 * i + 1]);
        }
      }
    } else if constexpr (FMT == kQ6K) {
      // nibbles: ql bytes 64 (G / 2) .., 32 per half; the upper halves for odd G; top bits: qh bytes 32 (G / 2) ..
      uint32_t qh[8];
      RowBlock<FMT>::words(base + 128 + 32 * (G >> 1), qh);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint32_t ql[8];
        RowBlock<FMT>::words(base + 64 * (G >> 1) + 32 * h, ql);
        const int sn = 4 * (G & 1), st = 4 * (G & 1) + 2 * h;
#pragma unroll
        for (int i = 0; i < 8; i++)
          four<32, 0>(((ql[i] >> sn) & 0x0F0F0F0Fu) | ((qh[i] >> st) & 0x03030303u) * 16u, ot[16 * h + 2 * i],
                      ot[16 * h + 2 * i + 1]);
      }
    } else {
      const uint32_t at = base + 68 * G;  // two blocks of 34 bytes; the first one's words straddle two loaded ones
      uint32_t prev = lds32(at);
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const uint32_t next = lds32(at + 32 * h + 4 * i + 4);
          four<128, 0>((h ? next : __funnelshift_r(prev, next, 16)) ^ 0x80808080u, ot[16 * h + 2 * i], ot[16 * h + 2 * i + 1]);
          prev = next;
        }
    }
  }
};

// Scale and offset of a row's groups: value = s * 2^-8 u + b * 2^-8 (s and b carry the 2^8).
template <int FMT>
struct UnitScale {
  uint32_t base, scw[2], mnw[2];
  float d, dmin;
  __device__ __forceinline__ void open(uint32_t at) {
    base = at;
    if constexpr (has_offset(FMT)) {
      uint32_t h[4];
      lds128(base, h);
      d = 256.f * half_bits_to_f32(h[0]), dmin = 256.f * half_bits_to_f32(h[0] >> 16);
      q4k_unpack_scales(h[1], h[2], h[3], scw[0], scw[1], mnw[0], mnw[1]);
    }
    if constexpr (FMT == kQ6K) d = 256.f * half_bits_to_f32(lds32((base + 208) & ~3u) >> ((base & 2) * 8));
  }
  __device__ __forceinline__ void group(int j, float& s, float& b) const {
    if constexpr (has_offset(FMT)) {
      s = d * (__uint_as_float((__byte_perm(scw[0], scw[1], j) & 0xFFu) | 0x4B000000u) - 8388608.f);
      const float m = dmin * (__uint_as_float((__byte_perm(mnw[0], mnw[1], j) & 0xFFu) | 0x4B000000u) - 8388608.f);
      b = fmaf(s, FMT == kQ5K ? 16.f : 8.f, -m);
    } else if constexpr (FMT == kQ6K) {
      s = d * static_cast<float>(lds_s8(base + 192 + j)), b = 0.f;
    } else {
      const uint32_t at = base + (FMT == kQ8 ? 34 : 18) * j;
      s = 256.f * half_bits_to_f32(lds32(at & ~3u) >> ((at & 2) * 8)), b = 0.f;
    }
  }
};

// Value k of a weight row in global memory (2-byte aligned), by the formats' own arithmetic.
template <int FMT>
__device__ float weight_at(const uint8_t* row, int k) {
  const int v = k & 255, l = v & 31, j = v >> 5;
  auto half_at = [](const uint8_t* p) { return half_bits_to_f32(*reinterpret_cast<const unsigned short*>(p)); };
  if constexpr (FMT == kQ8 || FMT == kQ40) {
    const uint8_t* b = row + static_cast<size_t>(k >> 5) * (FMT == kQ8 ? 34 : 18);
    if (FMT == kQ8) return half_at(b) * static_cast<float>(static_cast<signed char>(b[2 + l]));
    return half_at(b) * static_cast<float>(((b[2 + (l & 15)] >> (l < 16 ? 0 : 4)) & 15) - 8);
  } else {
    const uint8_t* b = row + static_cast<size_t>(k >> 8) * row_sb_bytes(FMT);
    if constexpr (FMT == kQ6K) {
      const int h = j >> 2, p = j & 3;
      const int q = ((b[64 * h + 32 * (p & 1) + l] >> (p < 2 ? 0 : 4)) & 15) | ((b[128 + 32 * h + l] >> (2 * p)) & 3) << 4;
      return half_at(b + 208) * static_cast<float>(static_cast<signed char>(b[192 + (v >> 4)])) * static_cast<float>(q - 32);
    } else {
      const uint8_t* c = b + 4;  // 6-bit scales and mins
      const int sc = j < 4 ? c[j] & 63 : (c[j + 4] & 15) | c[j - 4] >> 6 << 4;
      const int mn = j < 4 ? c[j + 4] & 63 : c[j + 4] >> 4 | c[j] >> 6 << 4;
      int q = (b[(FMT == kQ5K ? 48 : 16) + 32 * (j >> 1) + l] >> (4 * (j & 1))) & 15;
      if (FMT == kQ5K) q |= ((b[16 + l] >> j) & 1) << 4;
      return half_at(b) * static_cast<float>(sc) * static_cast<float>(q) - half_at(b + 2) * static_cast<float>(mn);
    }
  }
}

// A result that came out as NaN although its token has infinities and no NaN.  The centred integer of a weight that is not zero
// may be zero, its two terms may differ in sign, and the lower pieces of an f32 infinity are NaN; infinity times the weights has a sign
// all the same, and finite activations do not change it.  False: the NaN stands.  (bf16 activations of formats without an offset
// need none of this: infinity times the integer is the plain product.)
template <int FMT, bool XF>
__device__ __forceinline__ bool sum_of_infinities(const void* x, const uint8_t* w_row, int K, float& sum) {
  bool any = false;
  sum = 0.f;
  for (int k = 0; k < K; k += 4) {
    float f[4];
    if (XF) {
      const float4 v = *reinterpret_cast<const float4*>(static_cast<const float*>(x) + k);
      f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
    } else {
      const uint2 v = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(x) + k);
      f[0] = __uint_as_float(v.x << 16), f[1] = __uint_as_float(v.x & 0xFFFF0000u);
      f[2] = __uint_as_float(v.y << 16), f[3] = __uint_as_float(v.y & 0xFFFF0000u);
    }
#pragma unroll 1
    for (int e = 0; e < 4; e++) {
      const float v = e == 0 ? f[0] : e == 1 ? f[1] : e == 2 ? f[2] : f[3];
      if (fabsf(v) < INFINITY) continue;
      if (v != v) return false;
      sum = fmaf(v, weight_at<FMT>(w_row, k + e), sum);
      if (sum != sum) return false;  // zero weights, or infinities of both signs
      any = true;
    }
  }
  return any;
}

__host__ __device__ constexpr int tile_row(int f, int lane) { return f == kQ6K ? 8 * (lane & 15) + (lane >> 4) : lane; }

// TT: tokens that the sums are kept of (4, 8, 16); the MMAs always take 16.
template <int FMT, bool XF, int TT>
__global__ void __launch_bounds__(threads_of(XF), 2)
qgemm_unit_kernel(void* __restrict__ y, int y_dtype, const void* __restrict__ x, const uint8_t* __restrict__ wq, int M, int N, int K,
                  int KS, int early, int* err_word, const __grid_constant__ CUtensorMap x_map,
                  const __grid_constant__ CUtensorMap w_map) {
  extern __shared__ __align__(1024) unsigned char smem_u[];
  __shared__ SharedU sh;
  constexpr int kSV = stage_vals(FMT), kXS = x_slots(XF), WST = w_slots(FMT);
  constexpr int kGroup = kSV / 4;                  // four groups per stage
  constexpr int kXVals = x_vals(XF), kPerSb = 256 / kSV, kPerX = kXVals / kSV;  // stages per super-block / activation slot
  constexpr uint32_t kXSlot = x_bytes(XF), kPiece = kTok * kXVals * 2, kSub = kTok * 128;  // kSub: 64 values
  constexpr uint32_t kPitch = slot_pitch(FMT), kWBytes = slot_bytes(FMT), kSums = kXVals * 2;
  constexpr uint32_t kWOff = kXS * kXSlot, kSumOff = kWOff + WST * kWBytes, kRecvOff = kSumOff + kXS * kSums,
                     kRestOff = kRecvOff + kRecvBytes;
  constexpr bool kRest = keeps_rest(FMT), kOwn = keeps_stages(FMT), kLook = XF || has_offset(FMT);
  constexpr uint32_t kACol = kStages * 64;
  static_assert(kACol + kStages * (kSV / 2) <= kTmemCols && kXS <= kMaxX && WST <= kMaxW, "plan");
  static_assert(kWOff % 1024 == 0, "alignment");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_raw = static_cast<uint32_t>(__cvta_generic_to_shared(smem_u));
  const uint32_t smem_base = (smem_raw + 1023u) & ~1023u;
  unsigned char* const tiles = smem_u + (smem_base - smem_raw);
  auto bar_of = [&](const unsigned long long& b) { return static_cast<uint32_t>(__cvta_generic_to_shared(&b)); };
  const uint32_t wfull = bar_of(sh.wfull[0]), wempty = bar_of(sh.wempty[0]), xfull = bar_of(sh.xfull[0]),
                 xempty = bar_of(sh.xempty[0]), sfull = bar_of(sh.sfull[0]), afull = bar_of(sh.afull[0]),
                 done = bar_of(sh.done[0]), dempty = bar_of(sh.dempty[0]), pfull = bar_of(sh.pfull);
  uint32_t krank = 0;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(krank));
  const int vblock = static_cast<int>(blockIdx.x) / KS, vgrid = static_cast<int>(gridDim.x) / KS;
  volatile int* abort_flag = &sh.abort_flag;
  const int w_tiles = (N + 127) / 128, t_tiles = (M + kTok - 1) / kTok, ntiles = w_tiles * t_tiles;
  const int nsb_all = K >> 8;
  const int sb0 = nsb_all * static_cast<int>(krank) / KS, nsb = nsb_all * (static_cast<int>(krank) + 1) / KS - sb0;
  const int my_tiles = vblock < ntiles ? (ntiles - vblock + vgrid - 1) / vgrid : 0;
  const int total_sb = my_tiles * nsb;
  auto tile_info = [&](int tile, int& m0, int& n0) {
    const int wt = tile / t_tiles;
    m0 = (tile - wt * t_tiles) * kTok, n0 = wt * 128;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < WST; s++) {
      tc_mbar_init(wfull + 8 * s, 1);
      tc_mbar_init(wempty + 8 * s, 12);
    }
    for (int s = 0; s < kXS; s++) {
      tc_mbar_init(xfull + 8 * s, 1);
      tc_mbar_init(xempty + 8 * s, (kPerX > 1 ? 2 : 1) + (has_offset(FMT) ? (XF ? 4 : 5) : 0));
      tc_mbar_init(sfull + 8 * s, 1);
    }
    for (int s = 0; s < kStages; s++) {
      tc_mbar_init(afull + 8 * s, 4);
      tc_mbar_init(done + 8 * s, 1);
      tc_mbar_init(dempty + 8 * s, 4);
    }
    tc_mbar_init(pfull, 1);
    sh.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 12) {
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(&sh.tmem_base));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // the other ranks' barriers exist before anything arrives on them: awaited before the exchange
  if (KS > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  const uint32_t tmem_base = sh.tmem_base;
  if (!(early && warp == 14)) {
    pdl_wait();
    pdl_open();
  }
  bool ok = true, met = KS == 1;  // met: the cluster's first barrier has been waited for

  if (warp < 8) {
    // ------------------------------------------------------------ integers -> tensor memory
    const int row = threadIdx.x & 127, wrow = tile_row(FMT, row), set = warp >> 2;
    const uint32_t a_lane = tmem_base + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + kACol + (kSV / 2) * set;
    const uint32_t ring = smem_base + kWOff + row * kPitch;
    const int s = set;  // a set of four warps keeps to one stage in tensor memory
    int ws = 0;
    uint32_t phase = 0, wphase = 0;
    for (int tile = vblock; tile < ntiles && ok; tile += vgrid) {
      int m0_, n0;
      tile_info(tile, m0_, n0);
      uint32_t skew = 0, row_at = ring;  // Q6_K: as in qgemm_tc2.cu
      if (FMT == kQ6K) {
        skew = static_cast<uint32_t>((static_cast<size_t>(n0 + wrow) * nsb_all + sb0) * 210) & 15u;
        if (((n0 + wrow) >> 3) >= (N >> 3)) row_at = smem_base + kWOff + (128 + (wrow & 7)) * kPitch;
      }
      for (int sb = 0; sb < nsb && ok; sb++) {
        ok = __all_sync(0xFFFFFFFFu, tc_wait(wfull + 8 * ws, wphase, abort_flag));
        if (!ok) break;
        UnitRow<FMT> r;
        r.open(row_at + ws * kWBytes + skew);
#pragma unroll 1
        for (int i = set; i < kPerSb; i += 2) {
          // the MMAs that read this stage one ring turn ago must have completed: a look ahead of the arithmetic
          const bool ready = tc_mbar_test(done + 8 * s, phase ^ 1);
          uint32_t ot[32];
          r.group64(i * (kSV / 64), ot);
          if (kSV == 64 && i >= kPerSb - 2) {
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(wempty + 8 * ws);
          }
          if (!__all_sync(0xFFFFFFFFu, ready)) ok = __all_sync(0xFFFFFFFFu, tc_wait(done + 8 * s, phase ^ 1, abort_flag));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          tmem_st32(a_lane, ot);
          if constexpr (kSV == 128) {
            r.group64(i * 2 + 1, ot);
            if (i >= kPerSb - 2) {  // the last of the packed bytes has been read
              __syncwarp();
              if (lane == 0) tc_mbar_arrive(wempty + 8 * ws);
            }
            tmem_st32(a_lane + 32u, ot);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(afull + 8 * s);
          phase ^= 1;
        }
        if (++ws == WST) ws = 0, wphase ^= 1;
        if (FMT == kQ6K) skew = (skew + 210) & 15u;
      }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  } else if (warp < 12) {
    // ------------------------------------------------------------ group sums -> y
    const int row = threadIdx.x - 256, wrow = tile_row(FMT, row);
    const uint32_t d_lane = tmem_base + (static_cast<uint32_t>(32 * (warp & 3)) << 16);
    const uint32_t ring = smem_base + kWOff + row * kPitch;
    auto agree = [&](bool mine_ok) {  // the four warps take the same decision: nobody is left alone at a named barrier
      uint32_t all_ok;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 1, 128, q;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(all_ok)
          : "r"(mine_ok ? 1u : 0u)
          : "memory");
      return all_ok != 0;
    };
    // Results that this thread has stored, of tokens first .. first + n - 1, when one of them is not finite.
    auto look_again = [&](int first, int n, int out) {
#pragma unroll 1
      for (int m = first; m < first + n && m < M; m++) {
        const size_t at = static_cast<size_t>(m) * N + out;
        float sum = load_one(y, at, y_dtype);
        if (sum != sum && sum_of_infinities<FMT, XF>(static_cast<const char*>(x) + static_cast<size_t>(m) * K * (XF ? 4 : 2),
                                                     wq + static_cast<size_t>(out) * nsb_all * row_sb_bytes(FMT), K, sum))
          store_one(y, at, y_dtype, sum);
      }
    };
    float4* const rest = reinterpret_cast<float4*>(tiles + kRestOff) + row;  // this thread's own
    int s = 0, ws = 0, xs = 0;
    uint32_t phase = 0, wphase = 0, xphase = 0;
    for (int tile = vblock; tile < ntiles && ok; tile += vgrid) {
      int m0, n0;
      tile_info(tile, m0, n0);
      float acc[TT];
#pragma unroll
      for (int t = 0; t < TT; t++) acc[t] = 0.f;
      uint32_t skew = 0, row_at = ring;
      if (FMT == kQ6K) {
        skew = static_cast<uint32_t>((static_cast<size_t>(n0 + wrow) * nsb_all + sb0) * 210) & 15u;
        if (((n0 + wrow) >> 3) >= (N >> 3)) row_at = smem_base + kWOff + (128 + (wrow & 7)) * kPitch;
      }
      for (int sb = 0; sb < nsb && ok; sb++) {
        if (has_offset(FMT))
          ok = wait2(wfull + 8 * ws, wphase, (XF ? xfull : sfull) + 8 * xs, xphase, abort_flag);
        else
          ok = tc_wait(wfull + 8 * ws, wphase, abort_flag);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        UnitScale<FMT> sc;
        sc.open(row_at + ws * kWBytes + skew);
        float sg[has_offset(FMT) ? 8 : 4];
        float part[TT];  // a super-block is summed by itself: a long chain of additions into one sum rounds more
        if constexpr (has_offset(FMT)) {
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(wempty + 8 * ws);
#pragma unroll
          for (int h = 0; h < 256 / kXVals; h++) {
            if (h > 0) {
              ok = __all_sync(0xFFFFFFFFu, tc_wait((XF ? xfull : sfull) + 8 * xs, xphase, abort_flag));
              if (!ok) break;
            }
            const float* sums = reinterpret_cast<const float*>(tiles + kSumOff + xs * kSums);
#pragma unroll
            for (int g = 0; g < kXVals / 32; g++) {
              float b;
              sc.group(h * (kXVals / 32) + g, sg[h * (kXVals / 32) + g], b);
#pragma unroll
              for (int t = 0; t < TT; t += 4) {
                const float4 v = *reinterpret_cast<const float4*>(sums + kTok * g + t);
                if (h == 0 && g == 0) {
                  mul2(part[t], part[t + 1], v.x, v.y, b);
                  mul2(part[t + 2], part[t + 3], v.z, v.w, b);
                } else {
                  fma2(part[t], part[t + 1], v.x, v.y, b);
                  fma2(part[t + 2], part[t + 3], v.z, v.w, b);
                }
              }
            }
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(xempty + 8 * xs);
            if (++xs == kXS) xs = 0, xphase ^= 1;
          }
          if (!ok) break;
        }
#pragma unroll
        for (int i = 0; i < kPerSb; i++) {
          const bool ready = tc_mbar_test(done + 8 * s, phase);
          if constexpr (!has_offset(FMT)) {
            float b;
#pragma unroll
            for (int g = 0; g < 4; g++) sc.group(4 * i + g, sg[g], b);
            if (i == kPerSb - 1) {
              __syncwarp();
              if (lane == 0) tc_mbar_arrive(wempty + 8 * ws);
            }
          }
          if (!__all_sync(0xFFFFFFFFu, ready)) ok = __all_sync(0xFFFFFFFFu, tc_wait(done + 8 * s, phase, abort_flag));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int first_g = has_offset(FMT) ? 4 * i : 0;
          constexpr int kAtOnce = TT > 8 ? 1 : TT > 4 ? 2 : 4;          // groups in registers
          constexpr int kChunk = kOwn && TT > 8 ? 8 : TT;  // tokens
#pragma unroll
          for (int t0 = 0; t0 < TT; t0 += kChunk) {
            float own[kChunk];  // the stage's sums
#pragma unroll
            for (int g0 = 0; g0 < 4; g0 += kAtOnce) {
              float v[kAtOnce][kChunk];
#pragma unroll
              for (int g = 0; g < kAtOnce; g++) tmem_ld<kChunk>(d_lane + 64u * s + kTok * (g0 + g) + t0, v[g]);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              if (t0 + kChunk == TT && g0 + kAtOnce == 4) {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc_mbar_arrive(dempty + 8 * s);
              }
#pragma unroll
              for (int g = 0; g < kAtOnce; g++)
#pragma unroll
                for (int t = 0; t < kChunk; t += 2) {
                  float* const to = kOwn ? own + t : part + t0 + t;
                  if (!has_offset(FMT) && (kOwn || i == 0) && g0 + g == 0)
                    mul2(to[0], to[1], v[g][t], v[g][t + 1], sg[0]);
                  else
                    fma2(to[0], to[1], v[g][t], v[g][t + 1], sg[first_g + g0 + g]);
                }
            }
            if constexpr (kOwn)
#pragma unroll
              for (int t = 0; t < kChunk; t++) part[t0 + t] = i == 0 ? own[t] : part[t0 + t] + own[t];
          }
          if (++s == kStages) s = 0, phase ^= 1;
        }
        if (!ok) break;
#pragma unroll
        for (int t = 0; t < TT; t++) {
          const float before = acc[t];
          acc[t] += part[t];
          if (kRest) part[t] -= acc[t] - before;  // what the addition has rounded off
        }
        if constexpr (kRest)
#pragma unroll
          for (int q = 0; q < TT / 4; q++) {
            float4 r = sb ? rest[128 * q] : make_float4(0.f, 0.f, 0.f, 0.f);
            r.x += part[4 * q], r.y += part[4 * q + 1], r.z += part[4 * q + 2], r.w += part[4 * q + 3];
            rest[128 * q] = r;
          }
        if (++ws == WST) ws = 0, wphase ^= 1;
        if (FMT == kQ6K) skew = (skew + 210) & 15u;
      }
      if (KS > 1) ok = agree(ok);  // a warp may have given up on its own; all four come here, once: one tile per CTA
      if (!ok) break;
      if constexpr (kRest)
#pragma unroll
        for (int t = 0; t < TT; t++) {
          const float r = reinterpret_cast<const float*>(rest + 128 * (t / 4))[t % 4];
          if (fabsf(r) < INFINITY) acc[t] += r;  // not behind a sum that is infinite
        }
      if (KS == 1) {
        if (n0 + wrow < N) {
#pragma unroll
          for (int t = 0; t < TT; t++)
            if (m0 + t < M) store_one(y, static_cast<size_t>(m0 + t) * N + n0 + wrow, y_dtype, acc[t]);
          if (kLook && !all_finite(acc, M - m0)) look_again(m0, TT, n0 + wrow);
        }
        continue;
      }
      // K split, one tile: rank r owns rows own * r ..; [source][token quad][row] of 16 bytes
      const int own = (128 + KS - 1) / KS, first = own * static_cast<int>(krank), mine = min(own, 128 - first);
      if (row == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(pfull),
                     "r"(static_cast<uint32_t>((KS - 1) * (mine > 0 ? mine : 0) * TT * 4))
                     : "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      met = true;
      const int owner = row / own;
      const uint32_t at = smem_base + kRecvOff + ((krank * (TT / 4)) * own + (row - owner * own)) * 16;
      if (owner != static_cast<int>(krank)) {
        const uint32_t peer = tc_peer_addr(at, owner), peer_bar = tc_peer_addr(pfull, owner);
#pragma unroll
        for (int q = 0; q < TT / 4; q++) st_async16(peer + q * own * 16, acc + 4 * q, peer_bar);
      } else {
#pragma unroll
        for (int q = 0; q < TT / 4; q++)
          *reinterpret_cast<float4*>(tiles + (at - smem_base) + q * own * 16) =
              make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
      }
      ok = agree(tc_wait_cluster(pfull, 0, abort_flag));
      if (!ok) break;
      for (int i = row; i < mine * (TT / 4); i += 128) {
        const int q = i / mine, l = i - q * mine, out = n0 + tile_row(FMT, first + l);
        // In rank order; Q6_K, where it shows, even and odd ranks by themselves (pairs of pairs in all formats took registers from the
        // loop above: 28672x5120, sixteen tokens, Q4_K 44.3 -> 48.2 us, Q6_K 71 -> 77).
        float f[4] = {0.f, 0.f, 0.f, 0.f}, odd[4] = {0.f, 0.f, 0.f, 0.f};
        for (int r = 0; r < KS; r += kRest ? 2 : 1) {
          const unsigned char* const part_r = tiles + kRecvOff + ((r * (TT / 4) + q) * own + l) * 16;
          const float4 p = *reinterpret_cast<const float4*>(part_r);
          f[0] += p.x, f[1] += p.y, f[2] += p.z, f[3] += p.w;
          if (kRest && r + 1 < KS) {
            const float4 p1 = *reinterpret_cast<const float4*>(part_r + (TT / 4) * own * 16);
            odd[0] += p1.x, odd[1] += p1.y, odd[2] += p1.z, odd[3] += p1.w;
          }
        }
        if (kRest)
#pragma unroll
          for (int t = 0; t < 4; t++) f[t] += odd[t];
        if (out < N) {
#pragma unroll
          for (int t = 0; t < 4; t++)
            if (m0 + 4 * q + t < M) store_one(y, static_cast<size_t>(m0 + 4 * q + t) * N + out, y_dtype, f[t]);
          if (kLook && !all_finite(f, M - m0 - 4 * q)) look_again(m0 + 4 * q, 4, out);
        }
      }
    }
  } else if (warp < 14) {
    // ------------------------------------------------------------ MMA issuers, each for every other stage
    if (elect_one()) {
      // D = f32, A = B = bf16, both K-major, N = 16, M = 128
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kTok >> 3) << 17) | (8u << 24);
      const int s = warp - 12;
      const uint32_t a = tmem_base + kACol + (kSV / 2) * s, d = tmem_base + 64u * s;
      uint32_t phase = 0, xphase = 0;
      int xs = kPerX > 1 ? 0 : s, part = kPerX > 1 ? s : 0;
      for (int q = s; q < total_sb * kPerSb && ok; q += 2) {
        ok = wait3(dempty + 8 * s, phase ^ 1, xfull + 8 * xs, xphase, afull + 8 * s, phase, abort_flag);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int p = XF ? 2 : 0; p >= 0; p--) {  // the smallest piece first: an accumulation cuts bits off the sum so far
          const uint32_t x_at = smem_base + xs * kXSlot + p * kPiece + part * (kSV / 64) * kSub;
#pragma unroll
          for (int j = 0; j < kSV / 16; j++) {  // 16 values each; four steps are one sub-tile of 64
            const uint64_t b = make_sw128_desc(x_at + (j >> 2) * kSub) + 2 * (j & 3);
            umma_bf16_ts(d + kTok * (j / (kGroup / 16)), a + 8u * j, b, idesc,
                         (p < (XF ? 2 : 0) || j % (kGroup / 16) > 0) ? 1u : 0u);
          }
        }
        umma_commit(done + 8 * s);
        if (part + 2 >= kPerX) umma_commit(xempty + 8 * xs);  // this warp's last stage of the slot
        phase ^= 1;
        part += 2;
        if (part >= kPerX) {  // one slot on, or two where a slot is one stage
          part = kPerX > 1 ? s : 0;
          xs += kPerX > 1 ? 1 : 2;
          if (xs >= kXS) xs -= kXS, xphase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == 14) {
    // ------------------------------------------------------------ copies: packed weights, token tiles behind them
    int ws = 0, xs = 0;
    uint32_t wphase = 0, xphase = 0;
    bool waited = !early;
    auto issue_x = [&](int q) {
      const int ti = q / nsb, sb = sb0 + q - ti * nsb;
      int m0, n0_;
      tile_info(vblock + ti * vgrid, m0, n0_);
      ok = __all_sync(0xFFFFFFFFu, tc_wait(xempty + 8 * xs, xphase ^ 1, abort_flag));
      if (!ok) return;
      if (elect_one()) {
        const uint32_t bar = xfull + 8 * xs;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kXSlot) : "memory");
#pragma unroll
        for (int u = 0; u < 4; u++)
          asm volatile(
              "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                  "r"(smem_base + xs * kXSlot + u * kSub),
              "l"(reinterpret_cast<uint64_t>(&x_map)), "r"(bar), "r"(sb * 256 + u * 64), "r"(m0)
              : "memory");
      }
      __syncwarp();
      if (++xs == kXS) xs = 0, xphase ^= 1;
    };
    // token tiles are asked for kLead super-blocks behind the weights, which so run as far ahead as their ring allows
    constexpr int kLead = XF ? 0 : (WST > kXS ? WST - kXS : 0);
    int x_next = 0;
    for (int w = 0; w < total_sb && ok; w++) {
      if (!waited && w == WST) {  // the ring is full of requests made ahead of the dependency
        pdl_wait();
        pdl_open();
        waited = true;
      }
      if (!XF && waited)
        while (ok && x_next + kLead < w) issue_x(x_next++);
      if (!ok) break;
      const int ti = w / nsb, sb = sb0 + w - ti * nsb;
      int m0_, n0;
      tile_info(vblock + ti * vgrid, m0_, n0);
      ok = __all_sync(0xFFFFFFFFu, tc_wait(wempty + 8 * ws, wphase ^ 1, abort_flag));
      if (!ok) break;
      const uint32_t bar = wfull + 8 * ws, dst = smem_base + kWOff + ws * kWBytes;
      if constexpr (FMT == kQ6K) {  // groups of eight rows, see qgemm_tc2.cu
        const int groups = N >> 3;
        const int g0 = n0 >> 3, left = min(N - n0, 128) - 8 * min(groups - g0, 16);
        uint32_t extra = 0;
        size_t start = 0;
        int slot_row = 0;
        if (lane < left) {
          const size_t total = static_cast<size_t>(N) * nsb_all * 210, whole = total & ~static_cast<size_t>(15);
          const size_t o = (static_cast<size_t>(8 * groups + lane) * nsb_all + sb) * 210;
          start = o & ~static_cast<size_t>(15);
          size_t end = (o + 210 + 15) & ~static_cast<size_t>(15);
          slot_row = 128 + lane;
          if (end > whole) {
            end = whole;
            for (size_t b = whole; b < o + 210; b += 2)
              *reinterpret_cast<unsigned short*>(tiles + kWOff + ws * kWBytes + slot_row * kPitch + (b - start)) =
                  *reinterpret_cast<const unsigned short*>(wq + b);
          }
          extra = static_cast<uint32_t>(end - start);
        }
        const uint32_t boxes = g0 < groups ? 8u * 16u * kPitch : 0u;
        const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, extra) + boxes;
        __syncwarp();
        if (elect_one())
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(sum) : "memory");
        __syncwarp();
        if (boxes && elect_one())
          for (int b = 0; b < 8; b++)
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                    "r"(dst + b * 16 * kPitch),
                "l"(reinterpret_cast<uint64_t>(&w_map)), "r"(bar), "r"((((b * nsb_all + sb) * 210) & ~15) / 2), "r"(g0)
                : "memory");
        if (extra)
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                  dst + slot_row * kPitch),
              "l"(wq + start), "r"(extra), "r"(bar)
              : "memory");
      } else if (elect_one()) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kWBytes) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                dst),
            "l"(reinterpret_cast<uint64_t>(&w_map)), "r"(bar), "r"(static_cast<uint32_t>(sb) * kPitch / 2), "r"(n0)
            : "memory");
      }
      __syncwarp();
      if (++ws == WST) ws = 0, wphase ^= 1;
    }
    if (!waited) {
      pdl_wait();
      pdl_open();
    }
    if (!XF)
      while (ok && x_next < total_sb) issue_x(x_next++);
  } else if (!XF) {
    // ------------------------------------------------------------ activation sums of the groups (warp 15)
    if (has_offset(FMT)) {
      int xs = 0;
      uint32_t xphase = 0;
      const int mrow = lane & 15, mchunk = lane >> 4;  // ldmatrix: rows 0-15 of the first 16-byte column, then of the second
      for (int q = 0; q < total_sb && ok; q++) {
        ok = __all_sync(0xFFFFFFFFu, tc_wait(xfull + 8 * xs, xphase, abort_flag));
        if (!ok) break;
        float* sums = reinterpret_cast<float*>(tiles + kSumOff + xs * kSums);
#pragma unroll 4
        for (int g = 0; g < 8; g++) {
          float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int k = 0; k < 2; k++) {  // 16 values each
            const int chunk = 2 * (2 * (g & 1) + k) + mchunk;
            const uint32_t at = smem_base + xs * kXSlot + (g >> 1) * kSub + mrow * 128 + ((chunk ^ (mrow & 7)) << 4);
            uint32_t a[4];
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                         : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                         : "r"(at)
                         : "memory");
            const uint32_t unit = 0x3B803B80u;  // 2^-8
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %8}, "
                "{%0, %1, %2, %3};"
                : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(unit));
          }
          if ((lane & 3) == 0) {  // every column is the same sum
            sums[kTok * g + (lane >> 2)] = c[0];
            sums[kTok * g + 8 + (lane >> 2)] = c[2];
          }
        }
        __syncwarp();
        if (lane == 0) {
          tc_mbar_arrive(sfull + 8 * xs);
          tc_mbar_arrive(xempty + 8 * xs);
        }
        if (++xs == kXS) xs = 0, xphase ^= 1;
      }
    }
  } else if constexpr (XF) {
    // ------------------------------------------------------------ f32 tokens -> three swizzled bf16 tiles and the sums
    constexpr int kWarps = 2;
    static_assert(kXS == kWarps, "a warp keeps to one slot");
    const int xs = warp - 15;
    uint32_t xphase = 0;
    for (int q = xs; q < 2 * total_sb && ok; q += kWarps) {
      const int ti = (q >> 1) / nsb, sb = sb0 + (q >> 1) - ti * nsb;
      int m0, n0_;
      tile_info(vblock + ti * vgrid, m0, n0_);
      const int valid = min(kTok, M - m0);
      ok = __all_sync(0xFFFFFFFFu, tc_wait(xempty + 8 * xs, xphase ^ 1, abort_flag));
      if (!ok) break;
      const float* src = static_cast<const float*>(x) + static_cast<size_t>(m0) * K + sb * 256 + (q & 1) * 128;
      unsigned char* const slot = tiles + xs * kXSlot;
      float* sums = reinterpret_cast<float*>(tiles + kSumOff + xs * kSums);
#pragma unroll 2
      for (int i = 0; 2 * i < kTok; i++) {  // eight values of a token = one 16-byte unit per piece
        const int r = (lane >> 4) + 2 * i, u = lane & 15;
        if (2 * i >= valid) break;  // what lies there meets tokens that nobody stores
        float f[8];
        if (r < valid) {
          const float4* p = reinterpret_cast<const float4*>(src + static_cast<size_t>(r) * K + 8 * u);
          const float4 a = __ldg(p), b = __ldg(p + 1);
          f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
        } else {
#pragma unroll
          for (int e = 0; e < 8; e++) f[e] = 0.f;
        }
        if (has_offset(FMT)) {
          float g[8];
#pragma unroll
          for (int e = 0; e < 8; e++) g[e] = f[e] * 0x1p-8f;
          float t = ((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + (g[6] + g[7]));
          t += __shfl_xor_sync(0xFFFFFFFFu, t, 1);
          t += __shfl_xor_sync(0xFFFFFFFFu, t, 2);
          if ((u & 3) == 0) sums[kTok * (u >> 2) + r] = t;
        }
        uint32_t w[3][4];
#pragma unroll
        for (int e = 0; e < 4; e++) {  // upper 16 bits, twice, and the remainder
          const float a0 = f[2 * e], a1 = f[2 * e + 1];
          const uint32_t u0 = __float_as_uint(a0), u1 = __float_as_uint(a1);
          w[0][e] = __byte_perm(u0, u1, 0x7632);
          split_cut(a0 - __uint_as_float(u0 & 0xFFFF0000u), a1 - __uint_as_float(u1 & 0xFFFF0000u), w[1][e], w[2][e]);
        }
        const int off = (u >> 3) * static_cast<int>(kSub) + r * 128 + (((u & 7) ^ (r & 7)) << 4);
#pragma unroll
        for (int p = 0; p < 3; p++)
          *reinterpret_cast<uint4*>(slot + p * kPiece + off) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read through the async proxy
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(xfull + 8 * xs);
      xphase ^= 1;
    }
  }

  // ---- teardown: every role arrives here, whether it finished or gave up ----
  if (!met) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (KS > 1) tc_cluster_sync_relaxed();  // nobody leaves while another rank may still write here
  if (threadIdx.x == 0 && sh.abort_flag) report_device_error(err_word, UB_ERR_TIMEOUT);
  if (warp == 12) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// K split: the fewest super-blocks per CTA, an exchange counted as one, with all clusters resident at once.  Clusters of 1 .. 8
// CTAs that are, two CTAs per SM, as cudaOccupancyMaxActiveClusters reports them for 148 SMs.
inline int unit_split(int tiles, int nsb) {
  static const int most[9] = {0, 296, 148, 93, 71, 56, 45, 37, 33};
  const int slots = ub::num_sms() * 2;
  int best = 1, cost = (tiles + slots - 1) / slots * nsb;
  for (int ks = 2; ks <= 8 && ks <= nsb && tiles <= most[ks] * slots / 296; ks++)
    if ((nsb + ks - 1) / ks + 1 < cost) best = ks, cost = (nsb + ks - 1) / ks + 1;
  return best;
}

template <int FMT, bool XF, int TT>
int launch_unit(void* y, int y_dtype, const void* x, const void* wq, int M, int N, int K, bool fresh, cudaStream_t s) {
  constexpr size_t smem = smem_of(FMT, XF);
  static_assert(smem + sizeof(SharedU) + 1024 <= 114 * 1024, "two CTAs per SM");
  EncodeTiledFn enc = reinterpret_cast<EncodeTiledFn>(ub::tensor_map_encoder());
  if (!enc) return UB_ERR_UNSUPPORTED;
  const int tiles = ((N + 127) / 128) * ((M + kTok - 1) / kTok), slots = ub::num_sms() * 2, nsb = K / UB_QK_K;
  const int ks = unit_split(tiles, nsb);
  const int grid = ks > 1 ? tiles * ks : (tiles < slots ? tiles : slots);
  CUtensorMap xmap, wmap;
  memset(&xmap, 0, sizeof(xmap));
  memset(&wmap, 0, sizeof(wmap));
  const cuuint32_t estr[2] = {1, 1};
  if (!XF) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(M)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2};
    const cuuint32_t box[2] = {64, kTok};
    if (enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return UB_ERR_UNSUPPORTED;
  }
  {  // Q6_K: groups of eight rows, see qgemm_tc2.cu; 16-bit elements: a box may have at most 256 of them
    const int rows = FMT == kQ6K ? 8 : 1;
    const cuuint64_t bytes = static_cast<cuuint64_t>(nsb) * rows * row_sb_bytes(FMT);
    const cuuint64_t dims[2] = {bytes / 2, static_cast<cuuint64_t>(N >= rows ? N / rows : 1)};
    const cuuint64_t strides[1] = {bytes};
    const cuuint32_t box[2] = {slot_pitch(FMT) / 2, static_cast<cuuint32_t>(FMT == kQ6K ? 16 : 128)};
    if (enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(wq), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return UB_ERR_UNSUPPORTED;
  }
  auto kernel = qgemm_unit_kernel<FMT, XF, TT>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid), cfg.blockDim = dim3(threads_of(XF)), cfg.dynamicSmemBytes = smem, cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ks, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, kernel, y, y_dtype, x, static_cast<const uint8_t*>(wq), M, N, K,
                           ks, fresh ? 0 : 1, ub::device_error_word(), xmap, wmap);
  }
  if (e != cudaSuccess) {
    ub::set_cuda_error(e);
    return ub::fail(UB_ERR_CUDA);
  }
  return ub::check_launch();
}

template <int FMT, bool XF>
int by_tokens(void* y, int y_dtype, const void* x, const void* wq, int M, int N, int K, bool fresh, cudaStream_t s) {
  if (M <= 4) return launch_unit<FMT, XF, 4>(y, y_dtype, x, wq, M, N, K, fresh, s);
  if (M <= 8) return launch_unit<FMT, XF, 8>(y, y_dtype, x, wq, M, N, K, fresh, s);
  return launch_unit<FMT, XF, 16>(y, y_dtype, x, wq, M, N, K, fresh, s);
}

template <int FMT>
int by_type(void* y, int y_dtype, const void* x, bool x_f32, const void* wq, int M, int N, int K, bool fresh,
            cudaStream_t s) {
  return x_f32 ? by_tokens<FMT, true>(y, y_dtype, x, wq, M, N, K, fresh, s)
               : by_tokens<FMT, false>(y, y_dtype, x, wq, M, N, K, fresh, s);
}

// ---- up to sixteen tokens: this kernel, the decode kernels (CUDA cores, integer MMA) or two-piece weights (qgemm_tc2.cu) ----
// This kernel's time hardly depends on the tokens and falls with the matrix only down to the 3.5 us that the barriers, tensor
// memory and the cluster exchange take; a decode kernel's pass takes one, two, four or eight tokens and scales with the
// bytes.  No line of one size separates them, so all are priced, in us, by straight lines fitted to 23600 timings on B200 (256 to
// 16384 values, 300 to 28672 rows); nine of ten are within 15 %.  This kernel is taken where it is faster by more than a twentieth.  Some
// crossings, decode / this, bf16: Q4_K two tokens 14336x3328 10 / 14.5, four 4096x4352 18 / 8.5, four 14336x3328 14 / 16, eight
// 14336x3328 41 / 18; Q8_0 four tokens 6144x4096 9 / 10, four 6144x5120 76 / 12.5; Q6_K two tokens 1024x512 2.3 / 5.5, 28672x8192 69 / 92,
// 4096x14336 34 / 26; Q5_K one token 4096x14336 16.6 / 18.4, 8192x28672 450 / 54; Q4_0 one token 28672x8192 33 / 43, 4096x4352 24 / 8.
struct Pass {  // us: fixed, per super-block of a row, per 1024 rows, per both
  float fixed, sb, rows, sb_rows;
  float us(int N, int nsb) const {
    const float r = static_cast<float>(N) * (1.f / 1024.f);
    return fixed + sb * nsb + rows * r + sb_rows * nsb * r;
  }
};
constexpr float kNever = 1e9f;  // no decode kernel of this kind takes the pass

// Token passes as the dispatchers cut them.
float decode_us(int type, int M, int N, int K) {
  const int nsb = K / UB_QK_K;
  switch (type) {
    case 2:
    case 13:
    case 14: {  // one to four tokens: rows that are not whole 2048 values / staged, two CTAs per SM / one
      static const Pass lines[3][3][4] = {
          {{{1.206f, .544f, -.017f, .198f}, {1.209f, .88f, .004f, .236f}, {2.329f, 1.439f, .06f, .337f}, {1.578f, 1.127f, -.045f, .371f}},
           {{1.953f, .096f, .177f, .019f}, {1.786f, .18f, .164f, .037f}, {2.644f, .155f, -.073f, .088f}, {3.147f, .186f, -.05f, .103f}},
           {{1.075f, .099f, .17f, .027f}, {2.387f, .114f, .38f, .037f}, {1.46f, .222f, .716f, .042f}, {-.107f, .341f, 2.921f, -.031f}}},
          {{{1.165f, .627f, .017f, .242f}, {1.218f, .743f, .059f, .242f}, {2.418f, 1.305f, .09f, .436f}, {1.339f, 1.479f, -.243f, .477f}},
           {{2.196f, .039f, .189f, .036f}, {1.449f, .143f, .676f, .026f}, {1.841f, .208f, .326f, .073f}, {1.589f, .311f, .451f, .09f}},
           {{2.247f, .045f, .002f, .05f}, {3.245f, .06f, -.17f, .071f}, {2.218f, .135f, .799f, .082f}, {1.73f, .197f, 1.038f, .099f}}},
          {{{1.178f, .354f, .118f, .057f}, {1.341f, .406f, .156f, .076f}, {2.665f, .655f, .214f, .137f}, {1.482f, .494f, .212f, .107f}},
           {{1.616f, .084f, .564f, .013f}, {1.731f, .124f, .635f, .032f}, {2.036f, .181f, .356f, .066f}, {1.604f, .282f, .515f, .078f}},
           {{2.139f, .05f, -.006f, .053f}, {3.008f, .069f, -.123f, .072f}, {1.871f, .142f, .742f, .071f}, {1.897f, .188f, .945f, .093f}}}};
      const bool staged = type == 2 ? ub::q4_0_staged_takes(M, K) : type == 13 ? ub::q5k_staged_takes(M, K) : ub::q6k_staged_takes(M, K);
      if (M > 4 || (K % 2048 == 0 && !staged)) return kNever;
      return lines[type == 2 ? 0 : type == 13 ? 1 : 2][K % 2048 ? 0 : K <= 4096 ? 1 : 2][M - 1].us(N, nsb);
    }
    case 8: {
      static const Pass rest[4] = {{1.331f, .391f, .067f, .145f}, {1.181f, .594f, .027f, .244f}, {3.412f, .805f, .002f, .389f}, {1.196f, .987f, -.07f, .449f}};
      static const Pass lines[4] = {
          {.98f, .151f, .125f, .031f}, {1.88f, .144f, .08f, .037f}, {1.9f, .186f, .116f, .037f}, {2.45f, .343f, .146f, .049f}};
      if (K % 2048) return M <= 4 ? rest[M - 1].us(N, nsb) : kNever;
      float t = 0.f;
      for (int left = M, n; left > 0; left -= n) {
        n = left < 8 ? left : 8;
        if ((n > 4 ? 2 : 1) * (K / UB_QK8_0) > 568) return kNever;  // token quads in qgemv_imma.cu's shared memory
        t += lines[n == 1 ? 0 : n == 2 ? 1 : n <= 4 ? 2 : 3].us(N, nsb);
      }
      return t;
    }
    case 12: {
      static const Pass lines[4] = {
          {1.66f, .109f, .035f, .019f}, {1.25f, .186f, .038f, .02f}, {.74f, .353f, .041f, .03f}, {2.16f, .207f, .151f, .041f}};
      static const Pass odd[3] = {{2.87f, .031f, .166f, .021f}, {2.46f, .152f, .37f, .001f}, {3.f, .315f, .335f, .014f}};
      float t = 0.f;
      for (int left = M, n; left > 0; left -= n) {
        n = left < 8 ? left : 8;
        const bool made_for = K == 2048 || K == 4096 || (K == 8192 && n > 4);  // qgemv_mt.cu, qgemv_mc.cu
        if (!made_for && n > 1 && (n > 4 ? 4 : n > 2 ? 2 : 1) * nsb > 70) return kNever;  // token pairs, qgemv_imma.cu
        const int c = n == 1 ? 0 : n == 2 ? 1 : n <= 4 ? 2 : 3;
        if (c < 3) {
          t += (K % 2048 ? odd[c] : lines[c]).us(N, nsb);
        } else if (made_for) {
          t += lines[3].us(N, nsb);
        } else {  // tiles of 16 rows, four at a time between two reductions
          const int tiles = ((N + 15) / 16 + ub::num_sms() - 1) / ub::num_sms();
          t += 1.f + .36f * nsb + .88f * tiles + .065f * tiles * nsb + 2.5f * ((tiles + 3) / 4) + .046f * (n - 5) * nsb;
        }
      }
      return t;
    }
    default: return kNever;
  }
}

// us of a launch here: fixed, with a K split, per super-block of a CTA alone on its SM and of one of two.  Clusters fill SMs in
// pairs well before every SM has a CTA.
struct UnitCost {
  float fixed, split, one, two;
};
float unit_us(int type, int M, int N, int K, bool x_f32) {
  // up to four, eight, sixteen bf16 tokens, and f32 ones
  static const UnitCost costs[5][6] = {
      {{2.42f, 1.23f, .73f, 1.52f}, {2.79f, 1.4f, .79f, 1.61f}, {3.29f, 1.7f, 1.23f, 2.15f},
       {2.53f, 1.27f, 1.04f, 1.77f}, {2.89f, 1.09f, 1.79f, 2.57f}, {4.72f, .62f, 2.82f, 3.99f}},
      {{2.7f, 1.22f, .8f, 1.68f}, {2.26f, 1.38f, .89f, 1.68f}, {3.24f, 1.62f, .85f, 1.92f},
       {2.86f, 1.52f, .96f, 1.9f}, {2.57f, 1.1f, 1.65f, 2.54f}, {4.18f, .4f, 2.52f, 3.91f}},
      {{2.8f, 1.1f, .69f, 1.36f}, {2.97f, 1.22f, .63f, 1.37f}, {3.69f, 1.59f, .57f, 1.57f},
       {2.81f, 1.29f, .88f, 1.71f}, {2.6f, 1.25f, 1.48f, 2.3f}, {3.88f, .94f, 2.34f, 3.48f}},
      {{3.02f, 1.11f, .86f, 2.f}, {3.42f, .99f, .85f, 1.96f}, {4.09f, 1.14f, 1.17f, 2.51f},
       {2.94f, 1.24f, 1.01f, 2.25f}, {2.92f, 1.26f, 1.76f, 2.98f}, {4.83f, .67f, 2.82f, 4.34f}},
      {{3.29f, .94f, 1.41f, 2.83f}, {3.46f, .93f, 1.47f, 3.f}, {3.78f, 1.06f, 1.69f, 3.82f},
       {3.61f, 1.07f, 1.52f, 3.14f}, {3.83f, .55f, 1.9f, 3.66f}, {7.06f, -.95f, 2.76f, 4.83f}}};
  const UnitCost& c = costs[type == 12 ? 0 : type == 8 ? 1 : type == 2 ? 2 : type == 13 ? 3 : 4][(M <= 4 ? 0 : M <= 8 ? 1 : 2) + (x_f32 ? 3 : 0)];
  const int tiles = ((N + 127) / 128) * ((M + kTok - 1) / kTok), nsb = K / UB_QK_K, sms = ub::num_sms(), ks = unit_split(tiles, nsb);
  float us = c.fixed;
  if (ks > 1) {
    const float pairs = 2 * tiles * ks <= sms ? 0.f : tiles * ks <= sms ? .5f : 1.f;
    us += c.split + (nsb + ks - 1) / ks * (c.one + pairs * (c.two - c.one));
  } else {
    const int full = tiles / (2 * sms), left = tiles % (2 * sms);
    us += nsb * (full * c.two + (left == 0 ? 0.f : left <= sms ? c.one : c.two));
  }
  return us > 3.5f ? us : 3.5f;
}

// The same by the first fit (Q4_K, Q8_0; within 20 %): f32 results keep to the line that they were given, see few_tokens_route.
float unit_us_f32_results(int type, int M, int N, int K, bool x_f32) {
  static const UnitCost q4k[6] = {{-.94f, 4.18f, 1.04f, 1.62f}, {-.86f, 3.89f, 1.15f, 1.75f}, {.43f, 3.48f, 1.55f, 2.17f},
                                  {-1.1f, 4.09f, 1.41f, 1.95f}, {-1.42f, 4.33f, 2.25f, 2.71f}, {-2.42f, 6.1f, 3.66f, 4.33f}};
  static const UnitCost q8[6] = {{-.7f, 3.21f, 1.35f, 1.82f}, {-.69f, 3.28f, 1.37f, 1.85f}, {.42f, 3.f, 1.55f, 2.11f},
                                 {-.82f, 3.61f, 1.55f, 2.01f}, {-.85f, 3.32f, 2.2f, 2.68f}, {-1.09f, 4.58f, 3.45f, 4.27f}};
  const UnitCost& c = (type == 8 ? q8 : q4k)[(M <= 4 ? 0 : M <= 8 ? 1 : 2) + (x_f32 ? 3 : 0)];
  const int tiles = ((N + 127) / 128) * ((M + kTok - 1) / kTok), nsb = K / UB_QK_K, slots = ub::num_sms() * 2;
  const int ks = unit_split(tiles, nsb), ctas = ks > 1 ? tiles * ks : tiles;
  const int steps = ks > 1 ? (nsb + ks - 1) / ks : (tiles + slots - 1) / slots * nsb;
  const float us = c.fixed + (ks > 1 ? c.split : 0.f) + steps * (ctas > ub::num_sms() ? c.two : c.one);
  return us > 3.5f ? us : 3.5f;
}

// us of a launch with two-piece weights, up to sixteen tokens (within 10 %).
float two_piece_us(int type, int M, int N, int K, bool x_f32) {
  struct Cost {
    float fixed, step, step_f32;
  };
  const Cost c = type == 2    ? Cost{2.65f, 1.9f, 2.34f}
                 : type == 13 ? Cost{2.95f, 2.02f, 2.3f}
                 : type == 14 ? Cost{3.52f, 1.97f, 2.53f}
                 : type == 8  ? Cost{2.6f, 1.95f, 2.55f}
                              : Cost{2.4f, 1.77f, 2.2f};
  const int tiles = (N + 127) / 128, nsb = K / UB_QK_K, ks = ub::two_piece_split(tiles, nsb), sms = ub::num_sms();
  const int steps = (tiles * ks + sms - 1) / sms * ((nsb + ks - 1) / ks);
  return c.fixed + (ks > 1 ? 1.3f : 0.f) + (x_f32 ? c.step_f32 : c.step) * steps + .02f * M * (N * (1.f / 1024.f));
}

// Q4_K and Q8_0: are two-piece weights faster than the decode kernels, where those need a second pass or have the CUDA-core kernels' time?
// (f32 results stay with the CUDA-core kernels, which are the more exact ones.)
bool two_piece_pays(int type, int M, int N, int K, bool x_f32, bool y_f32) {
  const int pass = M < 8 ? M : 8, nsb = K / UB_QK_K;
  if (type == 8) {
    const bool quads_fit = K % 2048 == 0 && (pass + 3) / 4 * (K / UB_QK8_0) <= 568;  // in qgemv_imma.cu's shared memory
    if (quads_fit ? M <= 8 : y_f32) return false;
  } else {
    const bool made_for = K == 2048 || K == 4096 || (K == 8192 && M > 4);  // qgemv_mt.cu, qgemv_mc.cu
    const bool pairs_fit = (pass + 1) / 2 * nsb <= 70;  // token pairs of a whole row in qgemv_imma.cu's shared memory
    if (y_f32 && !made_for && !pairs_fit) return false;
    if (M <= 8 && (made_for || (M <= 4 && pairs_fit))) return false;
  }
  return 1.06f * two_piece_us(type, M, N, K, x_f32) < decode_us(type, M, N, K);
}

}  // namespace

namespace ub {

// Of 17300 calls of 1024 rows and values and more, timed without this kernel and with it, 200 take over 6 % longer with it: f32 results
// that are more exact for it, and crossings that the lines miss by a tenth.  With thresholds on the sizes there were 477.
//
// Q4_K and Q8_0, up to sixteen tokens: 0 the decode kernels, 1 this kernel, 2 two-piece weights (nine f32 tokens and more, where three
// pieces of an activation cost more than two of a weight: Q4_K sixteen tokens 8192x512 6.9 us there, 11.2 here).
// 16-bit results: the fastest, this kernel from a tenth on.  The rows that qgemv_mc.cu is made for stay there unless it takes 1.7 times as
// long (its bf16 result is its f32 one rounded).
// f32 results: the kernels differ by 2.7e-5 (activations of 15 bits) against 1e-7 here, so a call does not go back to
// the decode kernels for its time alone; where two-piece weights (2e-6 to 8e-6) would be faster than those, this kernel or they have
// the call.  From five tokens on the decode kernels' results have bits that other calls share (passes of eight tokens and the
// rest are two calls): they stay unless they take 1.7 times as long.
int few_tokens_route(int ggml_type, int M, int N, int K, bool x_f32, bool y_f32) {
  const bool two = M > 4 && two_piece_pays(ggml_type, M, N, K, x_f32, y_f32);
  const float decode = decode_us(ggml_type, M, N, K), unit = unit_us(ggml_type, M, N, K, x_f32);
  const float two_us = two && x_f32 && M > 8 ? two_piece_us(ggml_type, M, N, K, x_f32) : kNever;
  if (y_f32 && !(ggml_type == 8 && K % 2048)) {
    if ((M > 4 ? 1.7f : 1.05f) * unit_us_f32_results(ggml_type, M, N, K, x_f32) < decode) return 1;
    return !two ? 0 : two_us < unit ? 2 : 1;
  }
  if (two_us < unit && two_us < decode) return 2;
  const bool mc = ggml_type == 12 && M > 4 && M <= 8 && (K == 2048 || K == 4096 || K == 8192);
  return (mc ? 1.7f : 1.1f) * unit < decode ? 1 : 0;
}

// Q4_0, Q5_K and Q6_K: does this kernel take the call (instead of the staged kernels, qgemm_tc2.cu or the CUDA-core kernels)?
// f32 results of rows that the staged kernels take (15-bit activations, 2.7e-5) are this kernel's from where it was found the faster
// one at three shapes; they do not go back for their time alone (Q6_K two tokens 2048x10240 11.2 there, 17.4 here).  f32 results of
// one or two tokens of other Q6_K rows are the CUDA-core kernel's whatever the alignment of the weights.
// f32 results of more tokens: Q4_0 32 tokens 11520x8960 2450 / 55, Q6_K 182 tokens 14976x3584 1594 / 229.
bool unit_takes(int ggml_type, int M, int N, int K, bool x_f32, bool y_f32) {
  const bool odd = K % 2048 != 0;
  if (M > 16) return y_f32 && (odd || K > 4096);
  if (M > 4)  // two-piece weights otherwise; with bf16 activations they are never the faster ones
    return !(x_f32 && M > 8 && !y_f32) ||
           1.05f * unit_us(ggml_type, M, N, K, x_f32) < two_piece_us(ggml_type, M, N, K, x_f32);
  if (y_f32 && odd && ggml_type == 14 && M <= 2) return false;
  if (y_f32 && !odd) {
    if (ggml_type == 2) return M >= 3 || K > 8192 || (M >= 2 && K >= 4096);
    if (ggml_type == 13) return M >= 4 || K > 14336 || (M >= 2 && K >= 4096);
    return (M >= 2 && K > 8192) || (M >= 4 && K >= 4096);
  }
  return 1.05f * unit_us(ggml_type, M, N, K, x_f32) < decode_us(ggml_type, M, N, K);
}

// May a launch request weights ahead of its dependency wait?  Only where every kernel that could have the call does: a caller
// that writes weights with the kernel in front of a call which the plain launches take (CUDA-core kernels) needs no flag, and
// keeps its order here.  The decode kernels' first pass decides; where they do not take it, 16-bit results of Q4_K, Q8_0 and, from
// five tokens on, of the other formats were always requested ahead, except few tokens of Q8_0 rows that are not whole 2048
// values, which either kind took.
bool unit_early(int ggml_type, int M, int K, bool y_f32) {
  const bool odd = K % 2048 != 0;
  const int pass = ggml_type == 8 || ggml_type == 12 ? (M < 8 ? M : 8) : M < 4 ? M : 4;
  switch (ggml_type) {
    case 8: return q8_0_imma_takes(pass, K) || (!y_f32 && !(odd && (M <= 2 || M == 4)));
    case 12: return K == 2048 || K == 4096 || (K == 8192 && M > 4) || q4k_imma_takes(pass, K) || !y_f32;
    case 2: return !odd && (q4_0_staged_takes(pass, K) || (M > 4 && !y_f32));
    case 13: return !odd && (q5k_staged_takes(pass, K) || (M > 4 && !y_f32));
    default: return !odd && (q6k_staged_takes(pass, K) || (M > 4 && !y_f32));
  }
}

// K % 256 == 0, x and wq 16-byte aligned; UB_ERR_UNSUPPORTED (nothing launched, nothing recorded) for the rest and for
// formats and drivers it does not take.
int gguf_gemm_unit(int ggml_type, void* y, int y_dtype, const void* x, bool x_f32, const void* wq, int M, int N, int K,
                   bool fresh, cudaStream_t s) {
  if (M <= 0 || N <= 0 || K <= 0 || K % UB_QK_K || (reinterpret_cast<uintptr_t>(wq) & 15) ||
      (reinterpret_cast<uintptr_t>(x) & 15))
    return UB_ERR_UNSUPPORTED;
  if (!unit_early(ggml_type, M, K, y_dtype == UB_DTYPE_F32)) fresh = true;
  switch (ggml_type) {
    case 2: return by_type<kQ40>(y, y_dtype, x, x_f32, wq, M, N, K, fresh, s);
    case 8: return by_type<kQ8>(y, y_dtype, x, x_f32, wq, M, N, K, fresh, s);
    case 12: return by_type<kQ4K>(y, y_dtype, x, x_f32, wq, M, N, K, fresh, s);
    case 13: return by_type<kQ5K>(y, y_dtype, x, x_f32, wq, M, N, K, fresh, s);
    case 14: return by_type<kQ6K>(y, y_dtype, x, x_f32, wq, M, N, K, fresh, s);
    default: return UB_ERR_UNSUPPORTED;
  }
}

}  // namespace ub
