// Matmul of quantized weights on the tensor cores (tcgen05 / TMEM) at the precision of the decode kernels.
//
//   y[M,N] (f32 / bf16 / f16) = x[M,K] (bf16 or f32) . dequant(Wq)^T,   f32 accumulation
//
// The reference declares these block formats (kernels/quant.cpp:64-178) and multiplies dequantised copies
// (kernels/matmul.cpp:1143-1184).  The decode kernels here compute with exact weights and 15-bit activations; one
// bf16 operand would keep 8 bits of a weight.  So every weight is the sum of TWO bf16 values: w = d * scale * q - min is
// computed in f32, the first piece is w rounded to bf16 and the second the remainder rounded to bf16 (together within
// 2^-18 of w), and each K step multiplies the token tile by both.  f32 activations are split too (upper 16 bits and the
// remainder, which no magnitude overflows; within 2^-16); their product takes three MMAs (hi.hi, lo.hi, hi.lo), the
// fourth is below 2^-16 of a term and of either sign.  Error against f64, 2-norm of f32 results: 2e-6 to 5e-6, with f32
// activations 4e-6 to 1.2e-5 (rounding the first piece instead: 3.5e-6, but the second conversion per pair made 333
// tokens through 4096x4096 159 us instead of 108).
//
// One CTA per SM, tiles of 128 weight rows x up to TOK tokens, K in steps of 64 values:
//   warp 0        one lane issues tcgen05.mma (A from tensor memory, B from shared memory) and tcgen05.commit
//   warps 1-4     epilogue: accumulator -> y, or to the owning CTA of a K split
//   warps 5-12    dequantise: a thread owns one weight row (= TMEM lane) and one 32-value half of a step
//   warp 13       copies: packed weights of one super-block column (256 values of 128 rows) and bf16 token tiles
//   warps 14-17   (f32 activations) split the token tile into its two pieces
// Packed weights come as one tensor-map box per super-block column where rows are whole 16-byte pieces (all formats but
// Q6_K).  The 210-byte blocks of Q6_K put most rows off a 16-byte boundary; eight rows together are whole 16-byte pieces
// whatever the row length, so that matrix is viewed as N / 8 groups of eight rows and a column of 128 rows is eight boxes,
// box b = row b of sixteen groups, 240 bytes from the 16-byte boundary in front of the block.  The thread that reads a row
// knows the offset.  The up to seven rows behind the last whole group come by one bulk copy each.  (One bulk copy per row
// for all of them: 50 ns each, 6.4 us per super-block, 94 us for 4096x14336.)
//
// K split.  A tile may belong to a cluster of up to eight CTAs, each with a part of K.  When a CTA's MMAs are done
// its stage ring is free; it says so to the others and then serves as the buffer in which they leave their partial sums
// of the tokens that this CTA owns (four tokens at a time, st.async counted in bytes on a barrier of the owner).  The
// owner adds the parts in rank order: deterministic.
//
// Every wait is bounded; on expiry the CTA records UB_ERR_TIMEOUT, all roles leave and TMEM is freed.
#include <string.h>

#include "rowblock.cuh"

namespace ub {
void* tensor_map_encoder();
}

namespace {

using namespace ub;

constexpr int kProdWarps = 8;
constexpr int kXWarps = 4;
constexpr int kMaxStg = 6, kMaxW = 4;
constexpr uint32_t kBK = 64;
constexpr int threads_of(bool xf, int sets) { return (6 + kProdWarps * sets + (xf ? kXWarps : 0)) * 32; }

constexpr size_t smem_of(int f, int tok, int stages, int wst, bool xf, int pieces) {
  return static_cast<size_t>(stages) * tok * 128 * (xf || pieces == 1 ? 2 : 1) +
         static_cast<size_t>(wst) * slot_bytes(f) + 1024;
}

struct Shared2 {
  unsigned long long full[kMaxStg], empty[kMaxStg], wfull[kMaxW], wempty[kMaxW];
  unsigned long long tfull, tempty;  // accumulator complete / drained
  unsigned long long ready, pfull;   // K split: the other ranks' rings are free / all partial sums are here
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(taddr)
               : "memory");
}
// 16 bytes into another CTA's shared memory, counted on a barrier of that CTA
__device__ __forceinline__ void peer_store_tx4(uint32_t peer_addr, const uint32_t* v, uint32_t peer_bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(peer_addr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(peer_bar)
      : "memory");
}

__device__ __forceinline__ void store_y(void* y, size_t at, int dtype, float v) {
  if (dtype == UB_DTYPE_F32)
    static_cast<float*>(y)[at] = v;
  else if (dtype == UB_DTYPE_BF16)
    static_cast<__nv_bfloat16*>(y)[at] = __float2bfloat16_rn(v);
  else
    static_cast<__half*>(y)[at] = __float2half_rn(v);
}

// Row of the tile that a TMEM lane (= a row of a packed slot) holds.
__host__ __device__ constexpr int tile_row(int f, int lane) { return f == kQ6K ? 8 * (lane & 15) + (lane >> 4) : lane; }

// TOK: most tokens of a tile (64, 128, 256); tile_tok <= TOK: tokens a tile really takes (a multiple of 16).
// PIECES: 2 as described at the top.  1: weights rounded to bf16 once; a stage of 64 TMEM columns then holds 128 K values
// and two token sub-tiles of 64 values.
// CTAS: CTAs per SM (2: each takes half of the tensor and shared memory).
// SETS: sets of eight producer warps, each takes its part of the steps of every super-block.  Measured on B200, two pieces,
// 4096x14336: 30.5 us with two sets, 33.8 with one.
// UNR: unrolling of a set's steps: 2 for one piece (28672x4096, 16 tokens: 28.7 -> 26.5 us) and for Q6_K (4096x14336, five
// tokens: 36.8 -> 34.4 us), 1 for the others (Q4_K 30.5 / 31.8 us).  Handing a stage over only after the next one's
// arithmetic, as qgemm_tc.cu does, does not help here (26.5 / 27.9 us).
template <int FMT, int TOK, int STAGES, int WST, bool XF, int PIECES, int CTAS, int SETS, int UNR>
__global__ void __launch_bounds__(threads_of(XF, SETS), CTAS)
qgemm_tc2_kernel(void* __restrict__ y, int y_dtype, const float* __restrict__ xf, const uint8_t* __restrict__ wq, int M,
                 int N, int K, int tile_tok, int KS, int early, int* err_word, const __grid_constant__ CUtensorMap x_map,
                 const __grid_constant__ CUtensorMap w_map) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ __align__(1024) unsigned char smem2[];
  __shared__ Shared2 sh;
  static_assert(STAGES <= kMaxStg && WST <= kMaxW && TOK + 64 * STAGES <= 512 / CTAS, "plan");
  static_assert(PIECES == 2 || !XF, "f32 activations meet two-piece weights");
  constexpr int kSteps = PIECES == 2 ? 4 : 2;  // stages per super-block
  constexpr uint32_t kXBytes = TOK * 128, kStage = kXBytes * (XF || PIECES == 1 ? 2 : 1);
  constexpr uint32_t kPitch = slot_pitch(FMT), kWBytes = slot_bytes(FMT), kWOff = STAGES * kStage;
  static_assert(static_cast<uint32_t>(TOK) * 512 / 8 * 7 <= kWOff, "the ring takes the partial sums");
  constexpr uint32_t kACol = TOK, kTmemCols = 512 / CTAS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_raw = static_cast<uint32_t>(__cvta_generic_to_shared(smem2));
  const uint32_t smem_base = (smem_raw + 1023u) & ~1023u;
  unsigned char* const tiles = smem2 + (smem_base - smem_raw);
  const uint32_t bars = static_cast<uint32_t>(__cvta_generic_to_shared(&sh));
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (kMaxStg + s); };
  auto wfull_bar = [&](int s) { return bars + 8u * (2 * kMaxStg + s); };
  auto wempty_bar = [&](int s) { return bars + 8u * (2 * kMaxStg + kMaxW + s); };
  const uint32_t tfull_bar = bars + 8u * (2 * kMaxStg + 2 * kMaxW), tempty_bar = tfull_bar + 8, ready_bar = tfull_bar + 16,
                 pfull_bar = tfull_bar + 24;
  uint32_t krank = 0;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(krank));
  const int vblock = static_cast<int>(blockIdx.x) / KS, vgrid = static_cast<int>(gridDim.x) / KS;
  volatile int* abort_flag = &sh.abort_flag;
  const int w_tiles = (N + 127) / 128, t_tiles = (M + tile_tok - 1) / tile_tok, ntiles = w_tiles * t_tiles;
  const int nsb_all = K >> 8;
  const int sb0 = nsb_all * static_cast<int>(krank) / KS, nsb = nsb_all * (static_cast<int>(krank) + 1) / KS - sb0;
  auto tile_info = [&](int tile, int& m0, int& valid, int& n0) {
    const int wt = tile / t_tiles, tt = tile - wt * t_tiles;
    m0 = tt * tile_tok, valid = min(tile_tok, M - m0), n0 = wt * 128;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      tc_mbar_init(full_bar(s), kProdWarps + (XF ? kXWarps : 1));
      tc_mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < WST; s++) {
      tc_mbar_init(wfull_bar(s), 1);
      tc_mbar_init(wempty_bar(s), kProdWarps * SETS);
    }
    tc_mbar_init(tfull_bar, 1);
    tc_mbar_init(tempty_bar, 4);
    tc_mbar_init(ready_bar, KS > 1 ? KS - 1 : 1);
    tc_mbar_init(pfull_bar, 1);
    sh.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (KS > 1) tc_cluster_sync();  // the other ranks' barriers exist before anything arrives on them
  if (warp == 0) {
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(&sh.tmem_base));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = sh.tmem_base;
  const bool copy_warp = warp == 5 + kProdWarps * SETS;
  if (!(early && copy_warp)) asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp == 0) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      int s = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int tile = vblock; tile < ntiles && ok; tile += vgrid) {
        int m0_, valid, n0_;
        tile_info(tile, m0_, valid, n0_);
        const uint32_t n_mma = static_cast<uint32_t>((valid + 15) & ~15);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((n_mma >> 3) << 17) | (8u << 24);
        ok = tc_wait(tempty_bar, acc_phase ^ 1, abort_flag);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int ks = 0; ks < kSteps * nsb; ks++) {
          ok = tc_wait(full_bar(s), phase, abort_flag);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t bh = make_sw128_desc(smem_base + s * kStage);
          const uint32_t ah = tmem_base + kACol + 64u * s;
#pragma unroll
          for (int j = 0; j < 4; j++) umma_bf16_ts(tmem_base, ah + 8u * j, bh + 2 * j, idesc, (ks > 0 || j > 0) ? 1u : 0u);
          const uint64_t bl = make_sw128_desc(smem_base + s * kStage + kXBytes);  // second sub-tile
#pragma unroll
          for (int j = 0; j < 4; j++)
            umma_bf16_ts(tmem_base, ah + 32u + 8u * j, (PIECES == 2 ? bh : bl) + 2 * j, idesc, 1u);
          if (XF) {
#pragma unroll
            for (int j = 0; j < 4; j++) umma_bf16_ts(tmem_base, ah + 8u * j, bl + 2 * j, idesc, 1u);
          }
          umma_commit(empty_bar(s));
          if (++s == STAGES) s = 0, phase ^= 1;
        }
        if (!ok) break;
        umma_commit(tfull_bar);
        acc_phase ^= 1;
      }
    }
  } else if (warp <= 4) {
    // ------------------------------------------------------------ epilogue (TMEM lanes 32*(warp%4) ..)
    const int lane_base = 32 * (warp & 3), row = lane_base + lane, out_row = tile_row(FMT, row);
    const uint32_t acc = tmem_base + (static_cast<uint32_t>(lane_base) << 16);
    auto agree = [&](bool mine_ok) {  // the four warps take the same decision
      uint32_t all_ok;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 1, 128, q;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(all_ok)
          : "r"(mine_ok ? 1u : 0u)
          : "memory");
      return all_ok != 0;
    };
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int tile = vblock; tile < ntiles && ok; tile += vgrid) {  // with a K split: one tile at most
      int m0, valid, n0;
      tile_info(tile, m0, valid, n0);
      ok = agree(tc_wait(tfull_bar, acc_phase, abort_flag));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const bool live = n0 + out_row < N;
      const size_t at0 = static_cast<size_t>(m0) * N + n0 + out_row;
      if (KS == 1) {
#pragma unroll 1
        for (int c = 0; c < valid; c += 32) {
          uint32_t v[32];
          tmem_ld32(acc + c, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 32; j++)
            if (live && c + j < valid) store_y(y, at0 + static_cast<size_t>(c + j) * N, y_dtype, __uint_as_float(v[j]));
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(tempty_bar);
        acc_phase ^= 1;
        continue;
      }
      // K split: four tokens = one group, group g belongs to rank g % KS
      const int groups = (valid + 3) >> 2, slots = (groups + KS - 1) / KS;  // slots: groups a rank owns at most
      const int mine = (groups - static_cast<int>(krank) + KS - 1) / KS;
      if (warp == 1 && lane < KS && lane != static_cast<int>(krank))  // every MMA of this CTA has read the ring
        tc_peer_arrive(tc_peer_addr(ready_bar, static_cast<uint32_t>(lane)));
      if (warp == 1 && lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(pfull_bar),
                     "r"(static_cast<uint32_t>((KS - 1) * (mine > 0 ? mine : 0) * 2048))
                     : "memory");
      ok = agree(tc_wait_cluster(ready_bar, 0, abort_flag));
      if (!ok) break;
#pragma unroll 1
      for (int c = 0; c < valid; c += 32) {
        uint32_t v[32];
        tmem_ld32(acc + c, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const int g = (c >> 2) + q;
          const uint32_t owner = static_cast<uint32_t>(g) & (KS - 1);
          if (g < groups && owner != krank) {
            const uint32_t src = krank < owner ? krank : krank - 1;  // place of this rank among the owner's sources
            const uint32_t a = smem_base + ((src * slots + g / KS) * 128 + row) * 16;
            peer_store_tx4(tc_peer_addr(a, owner), v + 4 * q, tc_peer_addr(pfull_bar, owner));
          }
        }
      }
      ok = agree(tc_wait_cluster(pfull_bar, 0, abort_flag));
      if (!ok) break;
      for (int g = krank, i = 0; g < groups; g += KS, i++) {
        uint32_t own[4];
        tmem_ld4(acc + 4 * g, own);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        for (int r = 0; r < KS; r++) {
          float4 p = make_float4(__uint_as_float(own[0]), __uint_as_float(own[1]), __uint_as_float(own[2]),
                                 __uint_as_float(own[3]));
          if (r != static_cast<int>(krank))
            p = *reinterpret_cast<const float4*>(
                tiles + (((r < static_cast<int>(krank) ? r : r - 1) * slots + i) * 128 + row) * 16);
          f[0] += p.x, f[1] += p.y, f[2] += p.z, f[3] += p.w;
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (live && 4 * g + q < valid) store_y(y, at0 + static_cast<size_t>(4 * g + q) * N, y_dtype, f[q]);
      }
      break;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  } else if (warp <= 4 + kProdWarps * SETS) {
    // ------------------------------------------------------------ weights -> two bf16 pieces -> tensor memory
    const int tlane = 32 * (warp & 3) + lane;  // TMEM lane
    const int wrow = tile_row(FMT, tlane), half = ((warp - 5) >> 2) & 1, set = (warp - 5) >> 3;
    const uint32_t a_lane = tmem_base + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + kACol;
    const uint32_t ring = smem_base + kWOff + tlane * kPitch;
    constexpr int kOwn = kSteps / SETS;  // steps of a super-block that a set takes: kOwn * set, ...
    int s = kOwn * set, ws = 0;
    uint32_t phase = 0, wphase = 0;
    bool ok = true;
    for (int tile = vblock; tile < ntiles && ok; tile += vgrid) {
      int m0_, valid_, n0;
      tile_info(tile, m0_, valid_, n0);
      // Q6_K: where this row's first block starts inside its 16 bytes; the next one starts 210 bytes on
      uint32_t skew = 0;
      uint32_t row_at = ring;
      if (FMT == kQ6K) {
        skew = static_cast<uint32_t>((static_cast<size_t>(n0 + wrow) * nsb_all + sb0) * 210) & 15u;
        // rows behind the last whole group of eight have places of their own
        if (((n0 + wrow) >> 3) >= (N >> 3)) row_at = smem_base + kWOff + (128 + (wrow & 7)) * kPitch;
      }
      for (int sb = 0; sb < nsb && ok; sb++) {
        ok = __all_sync(0xFFFFFFFFu, tc_wait(wfull_bar(ws), wphase, abort_flag));
        if (!ok) break;
        RowBlock<FMT> blk;
        blk.open(row_at + ws * kWBytes + skew);
#pragma unroll UNR
        for (int i = 0; i < kOwn; i++) {
          const int step = kOwn * set + i;
          uint32_t hi[16], lo[16], group[32];
          if constexpr (PIECES == 2)
            blk.two_pieces(2 * step + half, hi, lo);
          else
            blk.one_piece(2 * step + half, group);  // half: which of the step's two 64-value groups
          if (i == kOwn - 1) {  // the last of the packed bytes has been read
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(wempty_bar(ws));
          }
          // the MMAs that read this stage one ring turn ago must have completed
          ok = __all_sync(0xFFFFFFFFu, tc_wait(empty_bar(s), phase ^ 1, abort_flag));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if constexpr (PIECES == 2) {
            tmem_st16(a_lane + 64u * s + 16u * half, hi);
            tmem_st16(a_lane + 64u * s + 32u + 16u * half, lo);
          } else {
            tmem_st32(a_lane + 64u * s + 32u * half, group);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(full_bar(s));
          if (++s == STAGES) s = 0, phase ^= 1;
        }
        if (SETS > 1) {  // the other set's steps
          s += kSteps - kOwn;
          if (s >= STAGES) s -= STAGES, phase ^= 1;
        }
        if (++ws == WST) ws = 0, wphase ^= 1;
        if (FMT == kQ6K) skew = (skew + 210) & 15u;
      }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  } else if (copy_warp) {
    // ------------------------------------------------------------ copies
    const int my_tiles = vblock < ntiles ? (ntiles - vblock + vgrid - 1) / vgrid : 0;
    const int total_sb = my_tiles * nsb;
    int s = 0, ws = 0, w_next = 0;
    uint32_t phase = 0, wphase = 0;
    bool ok = true;
    auto issue_w = [&]() {  // all lanes
      const int ti = w_next / nsb, sb = sb0 + w_next - ti * nsb;
      int m0_, valid_, n0;
      tile_info(vblock + ti * vgrid, m0_, valid_, n0);
      ok = __all_sync(0xFFFFFFFFu, tc_wait(wempty_bar(ws), wphase ^ 1, abort_flag));
      if (!ok) return;
      const uint32_t bar = wfull_bar(ws), dst = smem_base + kWOff + ws * kWBytes;
      if constexpr (FMT == kQ6K) {
        const int groups = N >> 3;  // of eight rows, all of them whole
        const int g0 = n0 >> 3, left = min(N - n0, 128) - 8 * min(groups - g0, 16);  // rows behind the last group: 0 .. 7
        // Rows behind the last group, one lane each.  The very last block of the matrix can end inside a 16-byte piece: its
        // copy stops at the piece before, the rest comes by 2-byte loads.
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
      w_next++;
      if (++ws == WST) ws = 0, wphase ^= 1;
    };
    for (int i = 0; i < WST - 1 && w_next < total_sb && ok; i++) issue_w();
    if (early) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int q = 0; q < total_sb && ok; q++) {
      if (w_next < total_sb) issue_w();
      if (!ok) break;
      if (XF) continue;
      const int ti = q / nsb, sb = sb0 + q - ti * nsb;
      int m0, valid_, n0_;
      tile_info(vblock + ti * vgrid, m0, valid_, n0_);
      for (int G = 0; G < kSteps; G++) {
        ok = __all_sync(0xFFFFFFFFu, tc_wait(empty_bar(s), phase ^ 1, abort_flag));
        if (!ok) break;
        if (elect_one()) {
          const uint32_t bar = full_bar(s);
          constexpr int kSub = 4 / kSteps;  // token sub-tiles of 64 values per stage
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                       "r"(static_cast<uint32_t>(tile_tok) * 128 * kSub)
                       : "memory");
#pragma unroll
          for (int u = 0; u < kSub; u++)
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                    "r"(smem_base + s * kStage + u * kXBytes),
                "l"(reinterpret_cast<uint64_t>(&x_map)), "r"(bar), "r"((sb * 4 + G * kSub + u) * static_cast<int>(kBK)),
                "r"(m0)
                : "memory");
        }
        __syncwarp();
        if (++s == STAGES) s = 0, phase ^= 1;
      }
    }
  } else if constexpr (XF) {
    // ------------------------------------------------------------ f32 tokens -> two swizzled bf16 tiles
    const int ct = threadIdx.x - (6 + kProdWarps * SETS) * 32;
    int s = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = vblock; tile < ntiles && ok; tile += vgrid) {
      int m0, valid, n0_;
      tile_info(tile, m0, valid, n0_);
      for (int ks = 0; ks < 4 * nsb && ok; ks++) {
        ok = __all_sync(0xFFFFFFFFu, tc_wait(empty_bar(s), phase ^ 1, abort_flag));
        if (!ok) break;
        const float* src = xf + static_cast<size_t>(m0) * K + (sb0 * 4 + ks) * static_cast<int>(kBK);
        unsigned char* const hi_t = tiles + s * kStage;
#pragma unroll 2
        for (int i = ct; i < valid * 8; i += kXWarps * 32) {  // eight values of a token row = one 16-byte unit per tile
          const int r = i >> 3, u = i & 7;
          const float4* p = reinterpret_cast<const float4*>(src + static_cast<size_t>(r) * K + 8 * u);
          const float4 a = __ldg(p), b = __ldg(p + 1);
          uint4 h, l;
          split_cut(a.x, a.y, h.x, l.x), split_cut(a.z, a.w, h.y, l.y);
          split_cut(b.x, b.y, h.z, l.z), split_cut(b.z, b.w, h.w, l.w);
          const int off = r * 128 + ((u ^ (r & 7)) << 4);  // 128-byte swizzle
          *reinterpret_cast<uint4*>(hi_t + off) = h;
          *reinterpret_cast<uint4*>(hi_t + kXBytes + off) = l;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read through the async proxy
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(full_bar(s));
        if (++s == STAGES) s = 0, phase ^= 1;
      }
    }
  }

  // ---- teardown: every role arrives here, whether it finished or gave up ----
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (KS > 1) tc_cluster_sync_relaxed();  // nobody leaves while another rank may still write or arrive here
  if (threadIdx.x == 0 && sh.abort_flag) report_device_error(err_word, UB_ERR_TIMEOUT);
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// The widest K split whose clusters are all resident at once.  A cluster stays inside one group of SMs.  Reported by
// cudaOccupancyMaxActiveClusters: with one CTA per SM 74 pairs, 33 clusters of four and 15 of eight, with two CTAs per SM
// 148, 71 and 33.  Sixteen of eight took a second round: Q6_K, five tokens, 2048 rows of 4096 values 19.8 us, with clusters
// of four 12.8.
inline int k_split(int tiles, int nsb, int ctas) {
  const int slots = ub::num_sms() * ctas, eights = ctas == 1 ? 15 : 16;
  int ks = 1;
  while (ks < 8 && nsb >= 4 * ks && tiles <= (ks == 1 ? slots / 2 : ks == 2 ? slots * 33 / 148 : slots * eights / 148))
    ks *= 2;
  return ks;
}

template <int FMT, int TOK, int STAGES, int WST, bool XF, int PIECES = 2, int CTAS = 1, int SETS = 2, int UNR = 1>
int launch2(void* y, int y_dtype, const void* x, const void* wq, int M, int N, int K, bool fresh, cudaStream_t s) {
  constexpr size_t smem = smem_of(FMT, TOK, STAGES, WST, XF, PIECES);
  static_assert(smem <= 226 * 1024 / CTAS, "shared memory plan");
  EncodeTiledFn enc = reinterpret_cast<EncodeTiledFn>(ub::tensor_map_encoder());
  if (!enc) return UB_ERR_UNSUPPORTED;
  // token tiles of equal size: 333 tokens are two tiles of 176, not 256 and 77
  const int t_tiles = (M + TOK - 1) / TOK, tile_tok = ((M + t_tiles - 1) / t_tiles + 15) / 16 * 16;
  const int tiles = ((N + 127) / 128) * t_tiles, slots = ub::num_sms() * CTAS, nsb = K / UB_QK_K;
  const int ks = k_split(tiles, nsb, CTAS);
  const int grid = ks > 1 ? tiles * ks : (tiles < slots ? tiles : slots);
  CUtensorMap xmap, wmap;
  memset(&xmap, 0, sizeof(xmap));
  memset(&wmap, 0, sizeof(wmap));
  const cuuint32_t estr[2] = {1, 1};
  if (!XF) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(M)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2};
    const cuuint32_t box[2] = {kBK, static_cast<cuuint32_t>(tile_tok)};
    if (enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return UB_ERR_UNSUPPORTED;
  }
  if (FMT == kQ6K) {  // groups of eight rows
    const cuuint64_t bytes = static_cast<cuuint64_t>(nsb) * 8 * row_sb_bytes(FMT);
    const cuuint64_t dims[2] = {bytes / 2, static_cast<cuuint64_t>(N >= 8 ? N / 8 : 1)};  // fewer than eight rows: not used
    const cuuint64_t strides[1] = {bytes};
    const cuuint32_t box[2] = {slot_pitch(FMT) / 2, 16};
    if (enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(wq), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return UB_ERR_UNSUPPORTED;
  } else {  // 16-bit elements: a box may have at most 256 of them, and a Q8_0 row piece is 272 bytes
    const cuuint64_t row_bytes = static_cast<cuuint64_t>(nsb) * row_sb_bytes(FMT);
    const cuuint64_t dims[2] = {row_bytes / 2, static_cast<cuuint64_t>(N)};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {row_sb_bytes(FMT) / 2, 128};
    if (enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(wq), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return UB_ERR_UNSUPPORTED;
  }
  auto kernel = qgemm_tc2_kernel<FMT, TOK, STAGES, WST, XF, PIECES, CTAS, SETS, UNR>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid), cfg.blockDim = dim3(threads_of(XF, SETS)), cfg.dynamicSmemBytes = smem, cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ks, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, kernel, y, y_dtype, static_cast<const float*>(x), static_cast<const uint8_t*>(wq), M, N, K,
                           tile_tok, ks, fresh ? 0 : 1, ub::device_error_word(), xmap, wmap);
  }
  if (e != cudaSuccess) {
    ub::set_cuda_error(e);
    return ub::fail(UB_ERR_CUDA);
  }
  return ub::check_launch();
}

template <int FMT>
int few(void* y, int y_dtype, const void* x, bool x_f32, const void* wq, int M, int N, int K, bool fresh, cudaStream_t s) {
  return x_f32 ? launch2<FMT, 64, 6, 3, true>(y, y_dtype, x, wq, M, N, K, fresh, s)
               : launch2<FMT, 64, 6, 4, false, 2, 1, 2, FMT == kQ6K ? 2 : 1>(y, y_dtype, x, wq, M, N, K, fresh, s);
}

template <int FMT>
int by_size(void* y, int y_dtype, const void* x, bool x_f32, const void* wq, int M, int N, int K, bool fresh,
            cudaStream_t s) {
  if (M <= 64) return few<FMT>(y, y_dtype, x, x_f32, wq, M, N, K, fresh, s);
  if (x_f32) return launch2<FMT, 128, 4, 2, true>(y, y_dtype, x, wq, M, N, K, fresh, s);
  if (M <= 128) return launch2<FMT, 128, 6, 3, false>(y, y_dtype, x, wq, M, N, K, fresh, s);
  return launch2<FMT, 256, 4, 2, false>(y, y_dtype, x, wq, M, N, K, fresh, s);
}

}  // namespace

namespace ub {

// K % 256 == 0, x and wq 16-byte aligned; UB_ERR_UNSUPPORTED (nothing launched, nothing recorded) for the rest and for
// formats and drivers it does not take.
int gguf_gemm_tc2(int ggml_type, void* y, int y_dtype, const void* x, bool x_f32, const void* wq, int M, int N, int K,
                  bool fresh, cudaStream_t s) {
  if (M <= 0 || N <= 0 || K <= 0 || K % UB_QK_K || (reinterpret_cast<uintptr_t>(wq) & 15) ||
      (reinterpret_cast<uintptr_t>(x) & 15))
    return UB_ERR_UNSUPPORTED;
  switch (ggml_type) {
    case 2: return by_size<kQ40>(y, y_dtype, x, x_f32, wq, M, N, K, fresh, s);
    case 13: return by_size<kQ5K>(y, y_dtype, x, x_f32, wq, M, N, K, fresh, s);
    case 14: return by_size<kQ6K>(y, y_dtype, x, x_f32, wq, M, N, K, fresh, s);
    // Q4_K and Q8_0: nine to sixteen f32 tokens, see few_tokens_route in qgemm_unit.cu
    case 12: return x_f32 && M <= 64 ? launch2<kQ4K, 64, 6, 3, true>(y, y_dtype, x, wq, M, N, K, fresh, s) : UB_ERR_UNSUPPORTED;
    case 8: return x_f32 && M <= 64 ? launch2<kQ8, 64, 6, 3, true>(y, y_dtype, x, wq, M, N, K, fresh, s) : UB_ERR_UNSUPPORTED;
    default: return UB_ERR_UNSUPPORTED;
  }
}

// Parts of K of a tile of 64 tokens.
int two_piece_split(int tiles, int nsb) { return k_split(tiles, nsb, 1); }

// y (bf16) = x (bf16) . W^T with weights rounded to bf16 once: the few-token launches of q4k_gemm_tc and q8_0_gemm_tc (fmt:
// GGML type; Q8_0 up to 64 tokens).  Two CTAs per SM up to 64 tokens of Q4_K: one CTA's chain of barriers (830 cycles per
// stage of 128 values, of which 500 are arithmetic) leaves the SM idle half of the time.  Measured on B200, us, against
// stages of 64 values in a kernel of its own (K split there too, even parts only): 16 tokens 28672x4096 38.5 -> 26.5,
// 57344x8192 129 -> 95, 8192x28672 58.6 -> 45.5; 100 tokens 4096x14336 84 -> 25 (no split there).  One CTA per SM with eight
// or sixteen producer warps: 36.5 and 36.8 for the first.
int q4k_gemm_tc1(int fmt, void* y, const void* x, const void* wq, int M, int N, int K, bool fresh, cudaStream_t s) {
  if (fmt == 8) return launch2<kQ8, 64, 6, 3, false, 1, 1, 1, 2>(y, UB_DTYPE_BF16, x, wq, M, N, K, fresh, s);
  if (M <= 64) return launch2<kQ4K, 64, 3, 3, false, 1, 2, 1, 2>(y, UB_DTYPE_BF16, x, wq, M, N, K, fresh, s);
  // more tokens: tiles of up to 128
  return launch2<kQ4K, 128, 4, 3, false, 1, 1, 1, 2>(y, UB_DTYPE_BF16, x, wq, M, N, K, fresh, s);
}

}  // namespace ub
