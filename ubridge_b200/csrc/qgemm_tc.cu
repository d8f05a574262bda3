// Prefill GEMM for Q4_K weights on the 5th-generation tensor cores (tcgen05 / TMEM), with the
// dequantisation fused into the main loop.
//
//   y[M,N] (bf16) = x[M,K] (bf16) . dequant(Wq[N rows of K/256 super-blocks])^T,   f32 accumulation.
//
// Replaces the reference's two-kernel sequence dequantize_block_q4_k_* (kernels/quant.cpp:477-488) +
// matmul_bf16 (kernels/matmul.cpp:1143-1184), whose W4 flavour dequantises a weight tile in on-chip memory
// and then calls the matrix engine (kernels/matmul.cpp:1039-1109).
//
// Tile and roles.  One persistent CTA per SM walks over (128 weight rows) x (TOK tokens) output tiles.
// The weight tile is the UMMA "A" operand (M = 128) and is read by the MMA from TENSOR MEMORY: producers
// dequantise straight from registers into TMEM with tcgen05.st, so weights never touch shared memory.
// The token tile is the "B" operand (N = TOK <= 256, trimmed to the valid tokens of a ragged last tile),
// K-major bf16 in the 128-byte-swizzled canonical layout, written to shared memory by 2-D tensor-map
// copies.  The accumulator D[128 lanes x TOK columns] lives in tensor memory next to the weight stages
// (columns 0..255 accumulators, 256.. weight stages of 64 columns each).  A weight stage holds 128 K values (two
// 64-value groups), a token stage 64; each token stage is four UMMA K=16 steps.
//
// What bounds it.  An MMA of 128 x 256 x 16 takes 128 cycles of the tensor pipe, a weight stage 1024.  A producer warp
// needs about 830 for it: 500 for the arithmetic of 64 values per thread and 75 to 150 for each barrier it looks at and for
// the stores to land, whatever they carry.  With stages of 64 values that chain was 700 cycles against 512 of MMAs: the
// producers held the tensor pipe back.  Weight stages of 128 values, one thread per 64-value group (both nibble halves from
// the same words), the issuing thread chosen by elect.sync and stores that land during the next stage's arithmetic took
// 2048 tokens at 14336x4096 from 190 to 177 us and 512 tokens at 57344x8192 from 376 to 335 us (bursts).  Dense launches
// of few tiles run in qgemm_tc2.cu (q4k_gemm_tc, q8_0_gemm_tc).
//
//   warp 0        allocates TMEM, then one elected lane issues tcgen05.mma and tcgen05.commit
//   warps 1-4     epilogue: tcgen05.ld -> bf16 -> staging tile in shared memory (accumulator released
//                 here) -> 16-byte coalesced stores to y, overlapping the next tile's main loop
//   warps 5-12    weight producers: read their row's packed super-block from a shared-memory ring, turn
//                 nibbles into the bf16 q * 2^-133 with one byte permute per pair, times d*sc minus dmin*m with
//                 packed bf16 FMAs (rowblock.cuh); tcgen05.st; the stage is handed over (tcgen05.wait::st, mbarrier
//                 arrive) after the next one's arithmetic
//   warp 13       one lane copies packed weight tiles ([128 rows][144 bytes], one 2-D tensor-map copy per super-block column)
//   warp 14       one lane copies token tiles (one copy per stage of 64 values)
//   Both as far ahead as their rings allow.  One thread for both took 650 cycles for a stage (a wait of 200 per barrier, 50 per
//   copy) and was what the grouped launches waited for.  With a thread for each, stages of the longest run's size instead of 128
//   tokens, runs that end with their last live token and looks at barriers one stage ahead, the expert layer of 256 tokens
//   (8 experts top-2, 4096 / 14336) takes 340 us instead of 399 (weights in one bf16 piece as in rowblock.cuh on both sides).
//
// Every mbarrier wait is bounded; on expiry the CTA sets a shared abort flag, records UB_ERR_TIMEOUT in
// the device error word, all roles leave their loops, and TMEM is freed before the kernel returns.
#include <string.h>

#include <mutex>

#include "rowblock.cuh"

namespace {

using namespace ub;

constexpr int kTcProducerWarps = 8;   // warps that dequantise a weight stage (128 rows x two 64-value groups)
constexpr int kTcThreads = (5 + kTcProducerWarps + 2) * 32;
constexpr int kTcBK = 64;

constexpr int kTcMaxStages = 8, kTcMaxAStages = 4;
constexpr int kTcWStages = 8;                        // most slots a ring of packed weight tiles has
// Shared-memory plan per token-tile size: the 256-token tile spends its memory on token stages (the
// copies' latency, not their bandwidth, bounds a K step) and keeps the other two areas small.
// With two CTAs per SM (the producer-bound MoE tiles of up to 128 tokens) every area is halved again.
// packed weight ring: WST slots when the launch names a depth, else 2 or 3
constexpr int tc_wstages(int tok, int ctas, int wst = 0) { return wst ? wst : ((tok > 128 || ctas > 1) ? 2 : 3); }
constexpr int tc_stage_tok(int tok, int ctas) {  // staging rows
  return (tok > 128 || ctas > 1) ? 64 : (tok < 128 ? tok : 128);
}
// Shared memory of a launch: token stages, output staging tile, packed-weight ring, 1 KB for alignment.
constexpr size_t tc_smem_bytes(int tok, int stages, int ctas, int wst, int fmt) {
  return static_cast<size_t>(stages) * (tok * 128) + static_cast<size_t>(tc_stage_tok(tok, ctas)) * 256 +
         static_cast<size_t>(tc_wstages(tok, ctas, wst)) * (128 * (fmt ? 8 * 34 : 144)) + 1024;
}
// One slot of the packed-weight ring holds 256 K values of 128 rows: a Q4_K super-block (144 bytes) or eight
// Q8_0 blocks (272 bytes, the shortest run of 34-byte blocks that is a whole number of 16-byte pieces).
constexpr uint32_t kTcQ8RowBytes = 8 * 34;
constexpr uint32_t tc_wrow(int fmt) { return fmt ? kTcQ8RowBytes : UB_Q4K_BYTES; }
constexpr uint32_t tc_wbytes(int fmt) { return 128 * tc_wrow(fmt); }

constexpr int kTcMaxRuns = 256;  // token runs (consecutive alignment blocks of one expert) a grouped launch handles

// Grouped (MoE) launch: rows of A are in aligned order (position i holds the token of sorted_ids[i]).
struct TcGroup {
  const int32_t* experts_ids;   // [blocks] expert of each alignment block, -1 = not on this rank
  const int32_t* num_post_pad;  // [1] padded number of positions
  const int32_t* sorted_ids;    // [positions] slot id (token * top_k + j) or a padding value >= num_valid
  const float* topk_w;          // [num_valid] routed weights (mode 2, may be null)
  int block;                    // alignment block size (multiple of 16, <= TOK)
  int num_valid;                // T * top_k
  int rows_per_expert;          // weight rows per expert in the packed tensor (2 I for mode 1, N for mode 2)
};

// Token tiles of one launch: dense, m[0] is the whole tile; grouped, m[i] is 32 (i + 1) tokens, so that a run of any length comes
// by one copy per stage (the copying thread issues some 50 cycles apart and waits 200 for each barrier).
struct TcXMaps {
  CUtensorMap m[4];
};

struct TcRun {
  int e, m0, len;
};

struct TcShared {
  unsigned long long full[kTcMaxStages], empty[kTcMaxStages];    // token stages
  unsigned long long afull[kTcMaxAStages], aempty[kTcMaxAStages];  // weight stages in tensor memory
  unsigned long long tmem_full[2], tmem_empty[2];
  unsigned long long wfull[kTcWStages], wempty[kTcWStages];
  uint32_t tmem_base;
  int abort_flag;
  int nruns, longest;
};

// TOK: tokens per tile (UMMA N): 64, 128 or 256.  STAGES: ring depth (token tiles in shared memory and
// weight stages in tensor memory advance together).
// MODE 0: dense y[M,N].  MODE 1 (grouped): weight tile = 64 gate rows + the 64 matching up rows of the run's
// expert, output act[position, N] = silu(gate) * up.  MODE 2 (grouped): output row sorted_ids[position],
// multiplied by the routed weight.  In the grouped modes M is the number of positions of A.
// CTAS: CTAs per SM the launch is planned for (2: each takes half of the SM's tensor memory and shared memory).
// WST: slots of the packed-weight ring (0: the default of tc_wstages).  Measured on B200: deeper rings do not
// help (MoE layer of 256 tokens, one CTA per SM: 3 -> 5 slots 589 -> 567 us; dense M = 2048: 2 -> 4 slots no
// change), the packed tiles are not what a K step waits for.
// FMT: 0 = Q4_K super-blocks, 1 = Q8_0 blocks (dense mode only).
// AST: weight stages in tensor memory.  One holds 128 K values (64 columns) and is written by the eight producer warps, a
// thread one 64-value group of its row; token stages hold 64 K values.
template <int TOK, int STAGES, int MODE, int CTAS, int WST, int FMT, int AST>
__global__ void __launch_bounds__(kTcThreads, CTAS)
qgemm_q4k_tc_kernel(__nv_bfloat16* __restrict__ y, int M, int N, int K, int* err_word,
                    const __grid_constant__ TcXMaps x_maps, const __grid_constant__ CUtensorMap w_map,
                    const TcGroup grp) {
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  __shared__ TcShared sh;
  __shared__ TcRun runs[MODE == 0 ? 1 : kTcMaxRuns];
  __shared__ float run_w[MODE == 2 ? TOK : 1];
  __shared__ int run_dst[MODE == 2 ? TOK : 1];
  // Looks at the next stage's barriers ahead of this one's work: the answer takes 200 cycles.  Grouped launches gain (below), with
  // 256 tokens of one tile nobody waits for it (2048 tokens 14336x4096 208 / 211 us).
  constexpr bool kLook = MODE != 0;
  static_assert(STAGES <= kTcMaxStages && (MODE == 0 || TOK <= 256), "barrier arrays");
  constexpr uint32_t kBBytes = TOK * 128;              // TOK token rows x 64 bf16
  constexpr int kStageTok = tc_stage_tok(TOK, CTAS);   // tokens the output staging tile holds
  constexpr int kWStages = tc_wstages(TOK, CTAS, WST);
  static_assert(kWStages <= kTcWStages, "barrier arrays");
  static_assert(FMT == 0 || MODE == 0, "the grouped modes take Q4_K experts");
  constexpr uint32_t kTcWBytes = tc_wbytes(FMT);
  constexpr uint32_t kWRow = tc_wrow(FMT);
  constexpr uint32_t kStagingOff = STAGES * kBBytes;   // [kStageTok tokens][128 weight rows] bf16
  constexpr uint32_t kWOff = kStagingOff + kStageTok * 256;  // packed weight ring: [128 rows][144 bytes] each
  constexpr int kAccBufs = (TOK > 128 || CTAS > 1) ? 1 : 2;  // accumulator buffers at the start of the allocation
  constexpr uint32_t kAccStride = 128;
  constexpr uint32_t kTmemCols = CTAS > 1 ? 256 : 512;        // columns this CTA allocates
  constexpr uint32_t kATmemCol = CTAS > 1 ? 128 : 256;        // first column of the weight stages (64 each)
  static_assert(TOK * kAccBufs <= static_cast<int>(kATmemCol) && kATmemCol + 64 * AST <= kTmemCols && AST <= kTcMaxAStages, "TMEM plan");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the swizzled tiles need 1024-byte alignment; the launch reserves 1 KB of slack for rounding the base up
  const uint32_t smem_raw = static_cast<uint32_t>(__cvta_generic_to_shared(tc_smem));
  const uint32_t smem_base = (smem_raw + 1023u) & ~1023u;
  unsigned char* const tiles = tc_smem + (smem_base - smem_raw);
  const uint32_t bars = static_cast<uint32_t>(__cvta_generic_to_shared(&sh));
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * kTcMaxStages + 8u * s; };
  auto afull_bar = [&](int b) { return bars + 16u * kTcMaxStages + 8u * b; };
  auto aempty_bar = [&](int b) { return afull_bar(kTcMaxAStages + b); };
  auto tfull_bar = [&](int b) { return afull_bar(2 * kTcMaxAStages + b); };
  auto tempty_bar = [&](int b) { return tfull_bar(2 + b); };
  auto wfull_bar = [&](int b) { return tfull_bar(4 + b); };
  auto wempty_bar = [&](int b) { return wfull_bar(kTcWStages + b); };
  const int vblock = static_cast<int>(blockIdx.x), vgrid = static_cast<int>(gridDim.x);
  volatile int* abort_flag = &sh.abort_flag;

  pdl_wait();
  pdl_open();
  constexpr int kTileCols = MODE == 1 ? 64 : 128;  // output columns per tile
  const int w_tiles = (N + kTileCols - 1) / kTileCols, t_tiles = (M + TOK - 1) / TOK;
  const int ksteps = K / (2 * kTcBK);

  if (MODE != 0) {
    // Token runs: consecutive alignment blocks of one expert, merged up to TOK tokens.  Every CTA builds
    // the same table (expert ids staged through the output staging tile, then one thread scans them).
    int* ids = reinterpret_cast<int*>(tiles + kStagingOff);
    const int padded = *grp.num_post_pad;
    int nblocks = padded > 0 ? (padded + grp.block - 1) / grp.block : 0;
    if (nblocks > kTcMaxRuns) nblocks = kTcMaxRuns;  // the launcher guarantees this never cuts
    for (int i = threadIdx.x; i < nblocks; i += kTcThreads) ids[i] = grp.experts_ids[i];
    __syncthreads();
    if (threadIdx.x == 0) {
      int n = 0;
      for (int b = 0; b < nblocks; b++) {
        const int e = ids[b];
        if (e < 0) continue;
        if (n > 0 && runs[n - 1].e == e && runs[n - 1].m0 + runs[n - 1].len == b * grp.block &&
            runs[n - 1].len + grp.block <= TOK) {
          runs[n - 1].len += grp.block;
        } else {
          runs[n].e = e, runs[n].m0 = b * grp.block, runs[n].len = grp.block;
          n++;
        }
      }
      sh.nruns = n, sh.longest = 1;
    }
    __syncthreads();
    // A run ends with its last live token, not with its last alignment block: what pads the block is neither read nor multiplied.
    for (int r = warp; r < sh.nruns; r += kTcThreads / 32) {
      int last = 0;
      for (int i = lane; i < runs[r].len; i += 32) {
        const int sid = grp.sorted_ids[runs[r].m0 + i];
        if (sid >= 0 && sid < grp.num_valid) last = i + 1;
      }
      last = __reduce_max_sync(0xFFFFFFFFu, last);
      if (lane == 0) runs[r].len = max(last, 1), atomicMax(&sh.longest, last);
    }
    __syncthreads();
  }
  // Token stages are as large as the longest run needs, and as many as fit: how far the copies run ahead is what a step of such a
  // launch waits for.
  constexpr bool kFit = MODE != 0 && TOK <= 128;
  const uint32_t x_stride = kFit ? static_cast<uint32_t>((sh.longest + 31) & ~31) * 128 : kBBytes;
  const int nst = kFit ? min(kTcMaxStages, static_cast<int>(STAGES * kBBytes / x_stride)) : STAGES;
  const int ntiles = MODE == 0 ? w_tiles * t_tiles : sh.nruns * w_tiles;
  // tile -> (first token row of A, valid tokens, first weight row in the packed tensor, first output column)
  auto tile_info = [&](int tile, int& m0, int& valid, int& wrow0, int& n0) {
    if (MODE == 0) {
      const int wt = tile / t_tiles, tt = tile - wt * t_tiles;
      m0 = tt * TOK, valid = min(TOK, M - m0), wrow0 = wt * 128, n0 = wt * 128;
    } else {
      const int run = tile / w_tiles, wt = tile - run * w_tiles;
      const TcRun r = runs[run];
      m0 = r.m0, valid = r.len, n0 = wt * kTileCols, wrow0 = r.e * grp.rows_per_expert + n0;
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kTcMaxStages; s++) {
      tc_mbar_init(full_bar(s), 1);
      tc_mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < AST; s++) {
      tc_mbar_init(afull_bar(s), kTcProducerWarps);
      tc_mbar_init(aempty_bar(s), 1);
    }
    for (int b = 0; b < 2; b++) {
      tc_mbar_init(tfull_bar(b), 1);
      tc_mbar_init(tempty_bar(b), 4);
    }
    for (int b = 0; b < kWStages; b++) {
      tc_mbar_init(wfull_bar(b), 1);
      tc_mbar_init(wempty_bar(b), kTcProducerWarps);
    }
    sh.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (warp == 0) {
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(&sh.tmem_base));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = sh.tmem_base;
  if (warp == 0) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      int s = 0, as = 0;
      uint32_t phase = 0, aphase = 0, acc_phase = 0;
      int buf = 0;
      bool ok = true, a_ready = false, x_ready = false;
      for (int tile = vblock; tile < ntiles && ok; tile += vgrid) {
        int m0_, valid, wrow0_, n0_;
        tile_info(tile, m0_, valid, wrow0_, n0_);
        // UMMA N = the tile's valid tokens rounded up to 16 (a ragged last tile costs less)
        const uint32_t n_mma = valid >= TOK ? TOK : static_cast<uint32_t>((valid + 15) & ~15);
        // instruction descriptor: D = f32, A = B = bf16, both K-major, N = n_mma, M = 128
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((n_mma >> 3) << 17) | (8u << 24);
        ok = tc_wait(tempty_bar(buf), acc_phase ^ 1, abort_flag);  // epilogue has drained this accumulator
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf) * kAccStride;
        for (int ks = 0; ks < ksteps; ks++) {
          if (!a_ready) ok = tc_wait(afull_bar(as), aphase, abort_flag);
          const uint32_t a_tmem = tmem_base + kATmemCol + 64u * as;
          const int as_next = as + 1 == AST ? 0 : as + 1;
          const uint32_t aphase_next = as_next ? aphase : aphase ^ 1;
#pragma unroll
          for (int g = 0; g < 2; g++) {
            if (ok && !x_ready) ok = tc_wait(full_bar(s), phase, abort_flag);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // looks at the next stages, ahead of this one's MMAs
            const int s_next = s + 1 == nst ? 0 : s + 1;
            const uint32_t phase_next = s_next ? phase : phase ^ 1;
            x_ready = kLook && tc_mbar_test(full_bar(s_next), phase_next);
            if (kLook && g == 1) a_ready = tc_mbar_test(afull_bar(as_next), aphase_next);
            const uint64_t b_desc = make_sw128_desc(smem_base + s * x_stride);
#pragma unroll
            for (int j = 0; j < 4; j++)  // K = 16 per instruction: 8 TMEM columns of A, 32 bytes of a B row
              umma_bf16_ts(d_tmem, a_tmem + 32u * g + 8u * j, b_desc + 2 * j, idesc, (ks > 0 || g > 0 || j > 0) ? 1u : 0u);
            umma_commit(empty_bar(s));  // stage is free once these MMAs have read it
            s = s_next, phase = phase_next;
          }
          if (!ok) break;
          umma_commit(aempty_bar(as));
          as = as_next, aphase = aphase_next;
        }
        if (!ok) break;
        umma_commit(tfull_bar(buf));  // accumulator complete
        if (++buf == kAccBufs) {
          buf = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else if (warp <= 4) {
    // ------------------------------------------------------------ epilogue (TMEM lanes 32*(warp%4) ..)
    const int lane_base = 32 * (warp & 3);
    const int ew = warp - 1;  // 0..3: which quarter of the tile's tokens this warp writes out
    unsigned char* const staging = tiles + kStagingOff;
    const bool vec_ok = (N % 8) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
    uint32_t acc_phase = 0;
    int buf = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
      int m0, valid, wrow0_, n0;
      tile_info(tile, m0, valid, wrow0_, n0);
      if (MODE == 2) {
        // destination row and routed weight of every token of the run (visible after the barrier below)
        for (int tk = threadIdx.x - 32; tk < valid; tk += 128) {
          const int sid = grp.sorted_ids[m0 + tk];
          const bool live = sid >= 0 && sid < grp.num_valid;
          run_dst[tk] = live ? sid : -1;
          run_w[tk] = live ? (grp.topk_w ? grp.topk_w[sid] : 1.f) : 0.f;
        }
      }
      {
        // all four epilogue warps take the same decision, so nobody is left alone at the named barrier
        const uint32_t mine = tc_wait(tfull_bar(buf), acc_phase, abort_flag) ? 1u : 0u;
        uint32_t all_ok;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 1, 128, q;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(all_ok)
            : "r"(mine)
            : "memory");
        ok = all_ok != 0;
      }
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // accumulator -> bf16 -> staging[token][weight row] -> y, kStageTok tokens at a time.  A warp's 32
      // lanes write 64 contiguous bytes of a staging row; token rows leave as 256 contiguous bytes.
      __nv_bfloat16* const st_col = reinterpret_cast<__nv_bfloat16*>(staging) + lane_base + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < valid; c0 += kStageTok) {
        const int part = min(kStageTok, valid - c0);
#pragma unroll 1
        for (int c = 0; c < part; c += 32) {
          uint32_t v[32];
          tmem_ld32(tmem_base + (static_cast<uint32_t>(lane_base) << 16) + static_cast<uint32_t>(buf) * kAccStride +
                        c0 + c, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 32; j++) {
            float f = __uint_as_float(v[j]);
            if (MODE == 2) f *= run_w[c0 + c + j];
            st_col[(c + j) * 128] = __float2bfloat16_rn(f);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("bar.sync 1, 128;" ::: "memory");  // the four epilogue warps: staging complete
        // after the last part the next tile's MMAs may overwrite the accumulator
        if (c0 + kStageTok >= valid && lane == 0) tc_mbar_arrive(tempty_bar(buf));
        if (MODE == 1) {
          // staging row = 64 gate values then 64 up values of one position: eight lanes per position
          const int ch = lane & 7;
          const bool n_in = n0 + 8 * ch < N;
          for (int t = 4 * ew + (lane >> 3); t < part; t += 16) {
            const uint4 gv = *reinterpret_cast<const uint4*>(staging + t * 256 + ch * 16);
            const uint4 uv = *reinterpret_cast<const uint4*>(staging + t * 256 + 128 + ch * 16);
            const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
            uint32_t ow[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const float g0 = __uint_as_float(gw[i] << 16), g1 = __uint_as_float(gw[i] & 0xFFFF0000u);
              const float u0 = __uint_as_float(uw[i] << 16), u1 = __uint_as_float(uw[i] & 0xFFFF0000u);
              const __nv_bfloat162 o2 =
                  __floats2bfloat162_rn(__fdividef(g0, 1.f + __expf(-g0)) * u0, __fdividef(g1, 1.f + __expf(-g1)) * u1);
              ow[i] = bf162_bits(o2);
            }
            if (n_in)
              *reinterpret_cast<uint4*>(y + static_cast<size_t>(m0 + c0 + t) * N + n0 + 8 * ch) =
                  make_uint4(ow[0], ow[1], ow[2], ow[3]);
          }
        } else if (vec_ok) {
          const int ch = lane & 15;
          const bool n_in = n0 + 8 * ch < N;
          for (int t = 2 * ew + (lane >> 4); t < part; t += 8) {
            const uint4 val = *reinterpret_cast<const uint4*>(staging + t * 256 + ch * 16);
            const int row = MODE == 2 ? run_dst[c0 + t] : m0 + c0 + t;
            if (n_in && row >= 0) *reinterpret_cast<uint4*>(y + static_cast<size_t>(row) * N + n0 + 8 * ch) = val;
          }
        } else {
          for (int t = ew; t < part; t += 4) {
            const int row = MODE == 2 ? run_dst[c0 + t] : m0 + c0 + t;
#pragma unroll
            for (int r = lane; r < 128; r += 32)
              if (n0 + r < N && row >= 0)
                y[static_cast<size_t>(row) * N + n0 + r] = reinterpret_cast<const __nv_bfloat16*>(staging)[t * 128 + r];
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");  // staging may be overwritten
      }
      if (++buf == kAccBufs) {
        buf = 0;
        acc_phase ^= 1;
      }
    }
  } else if (warp <= 4 + kTcProducerWarps) {
    // ------------------------------------------------------------ weight producers (256 threads per set)
    // One flat loop over (tile, super-block), two weight stages of 128 values each.  Packed weights arrive in shared memory
    // as [128 rows][144 bytes] per super-block; a thread owns one weight row (= its TMEM lane) and one of a stage's two
    // 64-value groups and reads its row's header and 32-byte pieces from there (rows are 144 bytes apart, so a
    // quarter-warp's 16-byte reads hit all 32 banks once).
    // weight row inside the tile = the TMEM lane this warp may access (32 * (warp % 4) + lane);
    // gsel: which group of a stage
    const int wrow = 32 * (warp & 3) + lane, gsel = (warp - 5) >> 2;
    const int nsb = K >> 8;
    const int my_tiles = vblock < ntiles ? (ntiles - vblock + vgrid - 1) / vgrid : 0;
    const int total_sb = my_tiles * nsb;  // super-block iterations
    const uint32_t w_ring = smem_base + kWOff + wrow * kWRow;
    const uint32_t a_lane = tmem_base + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + kATmemCol + 32u * gsel;

    int s = 0;  // weight stage being filled
    uint32_t phase = 0;
    int ws = 0;  // packed-weight ring slot
    uint32_t wphase = 0;
    bool ok = true;
    // A stage's stores land while the next one is computed; it is handed to the MMAs after that.
    int due = -1;
    auto hand_over = [&]() {
      if (due < 0) return;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(afull_bar(due));
      due = -1;
    };
    for (int q = 0; q < total_sb && ok; q++) {
      if (!__all_sync(0xFFFFFFFFu, tc_mbar_test(wfull_bar(ws), wphase))) {
        hand_over();
        ok = __all_sync(0xFFFFFFFFu, tc_wait(wfull_bar(ws), wphase, abort_flag));
        if (!ok) break;
      }
      RowBlock<FMT> blk;  // rows past N arrive as zeros: d = dmin = 0
      blk.open(w_ring + ws * kTcWBytes);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        // the MMAs that read this weight stage one ring turn ago must have completed: a look ahead of the arithmetic, whose
        // answer takes 120 cycles
        const bool ready = tc_mbar_test(aempty_bar(s), phase ^ 1);
        uint32_t ot[32];  // this thread's 64 values = 32 TMEM columns of packed pairs
        blk.one_piece(2 * i + gsel, ot);
        if (i == 1) {  // this warp has read all it needs from the slot
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(wempty_bar(ws));
        }
        hand_over();
        if (!__all_sync(0xFFFFFFFFu, ready)) ok = __all_sync(0xFFFFFFFFu, tc_wait(aempty_bar(s), phase ^ 1, abort_flag));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_st32(a_lane + 64u * s, ot);
        due = s;
        if (++s == AST) {
          s = 0;
          phase ^= 1;
        }
      }
      if (++ws == kWStages) {
        ws = 0;
        wphase ^= 1;
      }
    }
    hand_over();
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  } else if (warp == 5 + kTcProducerWarps) {
    // ------------------------------------------------------------ bulk copies of packed weights (one lane), as far ahead as
    // their ring allows
    if (elect_one()) {
      const int nsb = K >> 8;
      const int my_tiles = vblock < ntiles ? (ntiles - vblock + vgrid - 1) / vgrid : 0;
      const int total_sb = my_tiles * nsb;
      int ws = 0;
      uint32_t wphase = 0;
      bool ok = true;
      for (int q = 0; q < total_sb && ok; q++) {
        const int ti = q / nsb, sb = q - ti * nsb;
        int m0_, valid_, wrow0, n0_;
        tile_info(vblock + ti * vgrid, m0_, valid_, wrow0, n0_);
        ok = tc_wait(wempty_bar(ws), wphase ^ 1, abort_flag);
        if (!ok) break;
        const uint32_t bar = wfull_bar(ws);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kTcWBytes) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                "r"(smem_base + kWOff + ws * kTcWBytes),
            "l"(reinterpret_cast<uint64_t>(&w_map)), "r"(bar), "r"(sb * (FMT ? kWRow / 2 : kWRow)), "r"(wrow0)
            : "memory");
        if (MODE == 1)  // second half of the tile: the up rows matching the 64 gate rows (box = 64 rows)
          asm volatile(
              "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                  "r"(smem_base + kWOff + ws * kTcWBytes + kTcWBytes / 2),
              "l"(reinterpret_cast<uint64_t>(&w_map)), "r"(bar), "r"(sb * kWRow), "r"(wrow0 + N)
              : "memory");
        if (++ws == kWStages) {
          ws = 0;
          wphase ^= 1;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ bulk copies of token tiles (one lane), as far ahead of the
    // MMAs as their ring allows
    if (elect_one()) {
      const int nsb = K >> 8;
      const int my_tiles = vblock < ntiles ? (ntiles - vblock + vgrid - 1) / vgrid : 0;
      const int total_sb = my_tiles * nsb;
      int s = 0;
      uint32_t phase = 0;
      bool ok = true, x_ready = false;
      for (int q = 0; q < total_sb && ok; q++) {
        const int ti = q / nsb, sb = q - ti * nsb;
        int m0, valid, wrow0_, n0_;
        tile_info(vblock + ti * vgrid, m0, valid, wrow0_, n0_);
        const int box = MODE == 0 ? 0 : (valid - 1) >> 5;  // which map: no more tokens than the run has, in steps of 32
        const CUtensorMap* const x_map = &x_maps.m[TOK > 128 && MODE != 0 ? 3 : box];
        for (int G = 0; G < 4; G++) {
          if (!x_ready) ok = tc_wait(empty_bar(s), phase ^ 1, abort_flag);
          if (!ok) break;
          const int s_next = s + 1 == nst ? 0 : s + 1;
          const uint32_t phase_next = s_next ? phase : phase ^ 1;
          x_ready = kLook && tc_mbar_test(empty_bar(s_next), phase_next ^ 1);
          const uint32_t bar = full_bar(s);
          if (MODE != 0 && TOK > 128) {  // two boxes of 128 tokens at most
            const int boxes = (valid + 127) >> 7;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(boxes * 128 * 128) : "memory");
            for (int b = 0; b < boxes; b++)
              asm volatile(
                  "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                      "r"(smem_base + s * kBBytes + b * (128 * 128)),
                  "l"(reinterpret_cast<uint64_t>(x_map)), "r"(bar), "r"((sb * 4 + G) * kTcBK), "r"(m0 + 128 * b)
                  : "memory");
          } else {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                         "r"(MODE == 0 ? kBBytes : static_cast<uint32_t>((box + 1) * 32 * 128))
                         : "memory");
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                    "r"(smem_base + s * x_stride),
                "l"(reinterpret_cast<uint64_t>(x_map)), "r"(bar), "r"((sb * 4 + G) * kTcBK), "r"(m0)
                : "memory");
          }
          s = s_next, phase = phase_next;
        }
      }
    }
  }

  // ---- teardown: every role arrives here, whether it finished or gave up ----
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0 && sh.abort_flag) report_device_error(err_word, UB_ERR_TIMEOUT);
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// cuTensorMapEncodeTiled, resolved once through the runtime
EncodeTiledFn encode_tiled_fn() {
  static std::mutex mu;
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  std::lock_guard<std::mutex> lk(mu);
  if (!tried) {
    tried = true;
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

template <int TOK, int STAGES, int MODE, int CTAS = 1, int WST = 0, int FMT = 0>
int launch_tc(void* y, const void* x, const void* wq, int M, int N, int K, const TcGroup& grp, int w_rows_total,
              cudaStream_t s) {
  constexpr size_t smem = tc_smem_bytes(TOK, STAGES, CTAS, WST, FMT);
  constexpr int kAst = CTAS > 1 ? 2 : 4;
  static_assert(smem <= 227 * 1024 / CTAS, "shared memory plan");
  const int sms = ub::num_sms();
  int grid = sms * CTAS;  // grouped launches learn their tile count on the device; idle CTAs leave at once
  if (MODE == 0) {
    const int tiles = ((N + 127) / 128) * ((M + TOK - 1) / TOK);
    grid = tiles < sms ? tiles : sms;
  }
  // token matrix as a 2-D tensor map: inner dimension K (bf16), outer M; box = 64 x TOK, 128-byte swizzle;
  // rows beyond M read as zeros
  TcXMaps maps;
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return ub::fail(UB_ERR_UNSUPPORTED);
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(M)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2};
  const cuuint32_t estr[2] = {1, 1};
  memset(&maps, 0, sizeof(maps));
  for (int i = 0; i < (MODE == 0 ? 1 : 4); i++) {
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(MODE == 0 ? TOK : 32 * (i + 1))};
    if (enc(&maps.m[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return ub::fail(UB_ERR_UNSUPPORTED);
  }
  // packed weights as a 2-D byte tensor: inner dimension = one row's bytes, outer = all weight rows (of all
  // experts); box = one super-block (144 bytes) of 128 rows (64 for the gate/up halves of mode 1), no
  // swizzle; rows beyond the tensor read as zeros.  Q8_0: a box of eight blocks is 272 bytes, wider than the
  // 256 elements a box may have, so that map counts 16-bit elements (136 per box).
  CUtensorMap wmap;
  const cuuint64_t row_bytes = static_cast<cuuint64_t>(K / UB_QK_K) * tc_wrow(FMT);
  const cuuint64_t wdims[2] = {FMT ? row_bytes / 2 : row_bytes, static_cast<cuuint64_t>(w_rows_total)};
  const cuuint64_t wstrides[1] = {row_bytes};
  const cuuint32_t wbox[2] = {FMT ? tc_wrow(FMT) / 2 : tc_wrow(FMT), MODE == 1 ? 64u : 128u};
  if (enc(&wmap, FMT ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(wq), wdims,
          wstrides, wbox, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return ub::fail(UB_ERR_UNSUPPORTED);
  auto kernel = qgemm_q4k_tc_kernel<TOK, STAGES, MODE, CTAS, WST, FMT, kAst>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) {
    ub::set_cuda_error(e);
    return ub::fail(UB_ERR_CUDA);
  }
  return ub::launch_pdl_smem(kernel, dim3(grid), dim3(kTcThreads), smem, s, static_cast<__nv_bfloat16*>(y), M, N, K,
                             ub::device_error_word(), maps, wmap, grp);
}

// xg[i, :] = hidden[sorted_ids[i] / top_k, :] for the positions the alignment produced (padding is left as it is: the GEMMs
// store nothing of it)
__global__ void __launch_bounds__(256) moe_gather_rows_kernel(__nv_bfloat16* __restrict__ xg,
                                                              const __nv_bfloat16* __restrict__ hidden,
                                                              const int32_t* __restrict__ sorted_ids,
                                                              const int32_t* __restrict__ num_post_pad, int num_valid,
                                                              int top_k, int H) {
  const int i = blockIdx.x;
  pdl_wait();
  pdl_open();
  if (i >= *num_post_pad) return;
  const int sid = sorted_ids[i];
  if (sid < 0 || sid >= num_valid) return;
  const uint4* src = reinterpret_cast<const uint4*>(hidden + static_cast<size_t>(sid / top_k) * H);
  uint4* dst = reinterpret_cast<uint4*>(xg + static_cast<size_t>(i) * H);
  for (int c = threadIdx.x; c < H / 8; c += blockDim.x) dst[c] = __ldg(src + c);
}

}  // namespace

namespace ub {

// cuTensorMapEncodeTiled of the running driver as an untyped pointer (null when unavailable), for the other
// kernels of this library that build tensor maps.
void* tensor_map_encoder() { return reinterpret_cast<void*>(encode_tiled_fn()); }

// y (bf16) [M,N] = x (bf16) [M,K] . dequant(Wq)^T on tcgen05; K % 256 == 0, pointers 16-byte aligned.
// Returns UB_ERR_UNSUPPORTED when the driver offers no tensor-map encoder (the caller falls back).
int q4k_gemm_tc1(int fmt, void* y, const void* x, const void* wq, int M, int N, int K, bool fresh, cudaStream_t s);
int q4k_gemm_tc(void* y, const void* x, const void* wq, int M, int N, int K, bool fresh, cudaStream_t s) {
  // 128-token tiles (with a K split where they leave half of the SMs idle) while one round of CTAs holds all of them: 256-token
  // tiles would leave SMs without one.  Measured on B200, us, 128- / 256-token tiles: 4096 rows of 4096 values with 130
  // tokens 15.9 / 22.4, 256 18.8 / 27.1, 512 22.8 / 28.8; 4096x14336 with 200 tokens 37 / 63; 6144x4096 with 384 23.2 / 28.8.
  const int tiles128 = (N + 127) / 128 * ((M + 127) / 128);
  // (weights ahead of the dependency wait up to 64 tokens only: beyond, callers may have them written by the kernel in front)
  if (M <= 128 || tiles128 <= ub::num_sms()) return q4k_gemm_tc1(12, y, x, wq, M, N, K, fresh || M > 64, s);
  const TcGroup none = {nullptr, nullptr, nullptr, nullptr, 0, 0, 0};
  return launch_tc<256, 5, 0>(y, x, wq, M, N, K, none, N, s);
}

// Same product for Q8_0 rows (K/32 blocks of 34 bytes); K % 256 == 0 (a row must be whole 16-byte pieces) and wq
// 16-byte aligned, else UB_ERR_UNSUPPORTED and the caller keeps the decode kernel.  The 272-byte slots of the
// packed ring leave room for four token stages at 256 tokens.  No K split and 256-token tiles from 129 tokens on, however few
// tiles there are: the comparison with 128-token tiles on record (4096x4096, 512 tokens: 505 TFLOP/s against 400) is of
// producers that were slower by a fifth; the rule of q4k_gemm_tc has not been measured for this format.
int q8_0_gemm_tc(void* y, const void* x, const void* wq, int M, int N, int K, bool fresh, cudaStream_t s) {
  if (K % UB_QK_K || (reinterpret_cast<uintptr_t>(wq) & 15)) return UB_ERR_UNSUPPORTED;
  const TcGroup none = {nullptr, nullptr, nullptr, nullptr, 0, 0, 0};
  if (M <= 64) return q4k_gemm_tc1(8, y, x, wq, M, N, K, fresh, s);
  if (M <= 128) return launch_tc<128, 6, 0, 1, 2, 1>(y, x, wq, M, N, K, none, N, s);
  return launch_tc<256, 4, 0, 1, 0, 1>(y, x, wq, M, N, K, none, N, s);
}

// Limits of the grouped tcgen05 path; outside them the caller keeps the mma.sync kernels.
bool q4k_moe_tc_takes(int positions, int K, int N, int block) {
  return block > 0 && block % 16 == 0 && block <= 128 && K % UB_QK_K == 0 && N % 8 == 0 &&
         (positions + block - 1) / block <= kTcMaxRuns;
}
bool q4k_moe_tc_supported(int positions, int K, int N, int block) {
  return encode_tiled_fn() != nullptr && q4k_moe_tc_takes(positions, K, N, block);
}

// Gathers hidden rows into aligned order: xg[positions, H].
int moe_gather_rows(void* xg, const void* hidden, const int32_t* sorted_ids, const int32_t* num_post_pad, int positions,
                    int num_valid, int top_k, int H, cudaStream_t s) {
  if (positions <= 0) return UB_OK;
  return ub::launch_pdl(moe_gather_rows_kernel, dim3(positions), dim3(256), s, static_cast<__nv_bfloat16*>(xg),
                        static_cast<const __nv_bfloat16*>(hidden), sorted_ids, num_post_pad, num_valid, top_k, H);
}

// Grouped expert GEMM over rows in aligned order (A[positions, K] bf16).
//   act_silu_mul != 0: Bq = [E][2N rows: gate then up][K], C[position, N] = silu(gate) * up
//   else:              Bq = [E][N rows][K], C[sorted_ids[position], N] = (A . W^T) * topk_w[slot]
int q4k_moe_gemm_tc(void* C, const void* A, const void* Bq, const float* topk_w, const int32_t* sorted_ids,
                    const int32_t* experts_ids, const int32_t* num_post_pad, int positions, int K, int N, int E,
                    int num_valid, int block, int act_silu_mul, cudaStream_t s) {
  if (!q4k_moe_tc_supported(positions, K, N, block)) return UB_ERR_UNSUPPORTED;
  TcGroup g;
  g.experts_ids = experts_ids, g.num_post_pad = num_post_pad, g.sorted_ids = sorted_ids, g.topk_w = topk_w;
  g.block = block, g.num_valid = num_valid, g.rows_per_expert = act_silu_mul ? 2 * N : N;
  const int rows_total = E * g.rows_per_expert;
  // token runs are capped at the tile's token count: short runs (few tokens per expert) take the 128 tile
  const bool small = num_valid / (E > 0 ? E : 1) <= 128;
  if (act_silu_mul)
    return small ? launch_tc<128, 3, 1, 2>(C, A, Bq, positions, N, K, g, rows_total, s)
                 : launch_tc<256, 5, 1>(C, A, Bq, positions, N, K, g, rows_total, s);
  return small ? launch_tc<128, 3, 2, 2>(C, A, Bq, positions, N, K, g, rows_total, s)
               : launch_tc<256, 5, 2>(C, A, Bq, positions, N, K, g, rows_total, s);
}

}  // namespace ub
