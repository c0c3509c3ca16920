// FlashAttention forward for sm_100a.
//
// A block is G = 1 or 2 consecutive 128-row query tiles of one (batch, head) pair, whose key / value sequence is walked in
// 128-row tiles; one_tile_per_cta (fa_rules.h) says which G serves which call.  A CTA works on one block, or goes on with blocks that
// have not started (kTake, see take_over_pays): the producer asks for the next and publishes it, every role walks the same blocks.
// With G = 1 two CTAs share an SM.  Warp roles: G softmax groups, then four warps:
//   first    TMA producer (Q once per block, K/V ring; taking over: the next block)
//   second   tcgen05.mma issuer (d = 128: every product; d = 64: S = Q K^T only)
//   third    d = 64: second issuer, O += P V (two issuers keep S ahead)
//   fourth   padded batches: zeros in the output rows without a token; rows and padded batches: a look at the status word; else idle
// Tensor memory per query tile: 128 columns of fp32 scores S, D of fp32 output O, and at d = 64 64 of the 16-bit
// probabilities P, which feed the P*V product straight from tensor memory.  At d = 128 P overwrites the first 64
// columns of S; at d = 64 the next score product starts as soon as the group has read its scores.
//
// Softmax groups.  Quads (d = 64 beyond short sequences, and every call with dropout): eight warps per query tile, a warp owns 16 rows and
// a thread two of them with a quarter of their columns.  That is four softmax warps per scheduler; their work (per score
// element 8 clk of the exponential unit, about 5 instructions, 12 with dropout) overlaps where two warps
// per scheduler, each with a serial chain of waits, maxima and exponentials, fell into step and left the units idle
// for half of the time.  us, the four-warp groups before -> now: 8 x 12 x 4096 (d = 64) 526 -> 484, with dropout
// (ragged) 783 -> 616, 2 x 4 x 16384 causal 423 -> 383 (one tile per CTA at any length).  ncu, 8 x 12 x 2048 with
// dropout: issue slots busy 48 -> 63 %, 516 000 -> 404 000 clk.
// Rows (d = 128 without dropout, and short sequences): four warps per query tile, one thread per row.  At d = 128 the score product waits for P V
// of its own tile, two groups take turns on the tensor cores, and quads, whose group needs longer for a tile
// of its own, measured 8 % slower (4 x 12 x 8192 causal: 717 against 770 us).
//
// Numerics follow the reference forward (csrc/flash_attn/src/fmha_fprop_kernel_1xN.h:365-638):
// scores in fp32, p = exp2(scale*log2e*(s - max)), row sum of the un-dropped p, P rounded to the
// 16-bit input type before P*V, O accumulated in fp32 and scaled by 1/(sum * p_keep) at the end,
// LSE = max*scale + ln(sum), -inf for a row without any valid key.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstddef>
#include <type_traits>
#include "fa_kernels.h"
#include "fa_math.cuh"
#include "fa_rules.h"
#include "sm100_prims.cuh"

namespace fa {

namespace {

// G: query tiles (softmax groups) per CTA.  Two share every K / V tile, and one such CTA fills an SM.  One leaves
// room for a second CTA on the SM, whose loads, first products and epilogue run under the tiles of the other:
// for short sequences, where those are a third of a CTA's time (see one_tile_per_cta).
template <int D, int G, bool ROWS, bool TAKE = false>
struct FwdCfg {
  // Softmax layout.  Rows: a warpgroup per query tile, one thread per row.  Quads: eight warps per query tile, 16
  // rows each (see the softmax code for both).
  static constexpr bool kRows = ROWS;
  static constexpr int kGroupWarps = kRows ? 4 : 8;
  static constexpr int kSoftmaxWarps = G * kGroupWarps;
  static constexpr int kThreads = 32 * kSoftmaxWarps + 128;  // + 1 warpgroup (producer, MMA issuers, idle)
  // G = 1: 80 KB (d = 64: Q, two stages; 96 KB with a place for the output rows, kOutBytes) or 96 KB (d = 128: Q, one stage), so that
  // two CTAs fit
  static constexpr int kStages = (G == 1) ? ((D == 64) ? 2 : 1) : ((D == 64) ? 3 : 2);
  static constexpr int kPanels = D / 64;
  static constexpr int kTileBytes = kBlockM * D * 2;
  // Where the output rows pass through: Q's tile, or where a CTA goes on with another block (TAKE), whose Q is loaded ahead, a
  // place of their own, at d = 128 with one tile V's, which is needed last of the next block's operands.
  static constexpr bool kOutInV = TAKE && D == 128 && G == 1;  // (rows)
  static constexpr int kOutPiece = kOutInV ? kTileBytes / kSoftmaxWarps : ROWS ? 4096 : 2048;  // of a softmax warp
  static constexpr int kOutBytes = TAKE && !kOutInV && (ROWS || G == 1) ? kSoftmaxWarps * kOutPiece : 0;  // beside Q, K and V
  static constexpr int kSmemBytes = (G + 2 * kStages) * kTileBytes + kOutBytes + 1024;
  static constexpr uint32_t kTmemCols = 256 * G;
  static constexpr uint32_t kTmemS0 = 0, kTmemS1 = 128, kTmemO0 = 128 * G, kTmemO1 = 128 * G + D;
  // d = 64 leaves 128 tensor-memory columns free: P gets its own columns there, so the next
  // S = Q K^T can be issued as soon as the softmax group has read the current S into registers.
  // At d = 128 the 512 columns are full and P overwrites the first 64 columns of its S buffer.
  static constexpr bool kSeparateP = (D == 64);
  static constexpr uint32_t kTmemP0 = kSeparateP ? 192 * G : kTmemS0, kTmemP1 = kSeparateP ? 192 * G + 64 : kTmemS1;
  // register split (per thread) of the 128 or 168 (rows), 80 or 96 (quads) a thread is launched with
  static constexpr int kSoftmaxRegs = kRows ? ((G == 1) ? 208 : 224) : ((G == 1) ? 96 : 104);
  static constexpr int kOtherRegs = kRows ? ((G == 1) ? 48 : 56) : ((G == 1) ? 48 : 64);
  static constexpr uint32_t kArrivals = kRows ? 128 : 8;  // of a softmax group: every thread, or one lane per warp
  // Output rows straight from the registers instead of through shared memory.  Pairs of query tiles at d = 64 have sixteen softmax warps,
  // whose loop is the slower one beside the staged epilogue (a phase of the two groups or the registers: 0 instead of 64-80 bytes of spills).
  // us, staged -> now: 2 x 16384 and 3 x 1 tokens, 4 heads 697 -> 672, causal 372 -> 348, with dropout 1293 -> 1240, causal 683 -> 659;
  // 1 x 2048, 16 heads 34.8 -> 32.8; the other way round 4 x 700, 12 heads 20.5 -> 21.6.
  // Hence the columns that a warp of the epilogue stores by TMA at once, 0 for none; in quads a warp holds half of a row.
  static constexpr int kBoxRows = 64, kBoxQuads = D == 64 && G == 2 ? 0 : D / 2;
};

constexpr int kMaxSparseTiles = 1024;  // key tiles of 128 per sequence in block-sparse mode

// What a CTA works on: the query tiles [mp * G, mp * G + G) of one (batch, head) pair; n(g): key tiles of each.  mp < 0: behind the
// last block
struct FwdBlock {
  int q_start, sq, k_start, sk, h, b, mp, n0, n1;
  __device__ __forceinline__ int n(int g) const { return g == 0 ? n0 : n1; }  // (an array would go to local memory)
};

template <int STATS>
struct FwdShared {
  uint64_t q_full[2];
  uint64_t k_full[3], k_empty[3], v_full[3], v_empty[3];
  uint64_t s_full[2], s_free[2], p_half[2], p_full[2], o_full[2];
  uint64_t drained[2];  // of the two issuing warps, at their end
  // from here on: CTAs that take over blocks
  uint64_t q_empty[2];
  uint64_t next_full;                 // the answer to a request for another block is in `next`
  uint64_t blk_full[2], blk_done[2];  // the block after is in `blk`; every role has finished the one there
  uint64_t out_free;                  // the rows of a block have left the place they pass through
  uint64_t stats_full[2];             // a group's row statistics are written (bounded, unlike bar.sync)
  float2 row_stats[STATS][kBlockM];  // (max, sum) of every query row, for the epilogue; taking over: two of a group, by the block's parity
  alignas(16) uint4 next;
  FwdBlock blk[2];  // block k in entry k % 2
  uint32_t alive;   // pairs: changes as the producer gets on (see mbar_wait_alive)
  uint32_t tmem_base;
  int abort_flag;
  int stop;  // a CTA of this launch has abandoned a wait
};
constexpr int kBarriers = 26, kTakeBarriers = 36;  // at the head of FwdShared
static_assert(offsetof(FwdShared<1>, s_free) == 16 * 8 && offsetof(FwdShared<1>, o_full) == 22 * 8 && offsetof(FwdShared<1>, q_empty) == kBarriers * 8 && offsetof(FwdShared<1>, row_stats) == kTakeBarriers * 8, "order of the barriers");

template <int N>
__device__ __forceinline__ void reg_alloc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void reg_dealloc() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// Epilogue of 32 query rows (a warp, thread = row, 32x32b shape), NC 32-column groups from c0 on: O = acc / (sum * p_keep)
// in the 16-bit type; the warp of the first group also writes LSE = max * scale + ln(sum).  A row without any valid key
// gets zeros and -inf.  Out through `piece`, the warp's NC * 2048 bytes of shared memory (see stage_offset), in boxes of BOX columns;
// 0: from the registers.  ig: first query row of the warp.  REUSE: the piece holds one panel, and what was stored from it before
// (by lane 0) has to be read first; else this waits until its own stores have read it.
template <bool BF16, int NC, int BOX, bool REUSE>
__device__ __forceinline__ void store_rows(const KernelArgs& a, const CUtensorMap* tm_o, uint32_t tO, int c0, bool have_acc, bool ok, int ig, int lane,
                                           int sq, int q_start, int b, int h, float m_run, float l_run, uint8_t* piece) {
  constexpr bool STAGED = BOX != 0;
  constexpr int CH = STAGED ? BOX / 8 : 8;  // 16-byte chunks of a row in one panel of the piece
  static_assert(!STAGED || CH == (NC == 1 ? 4 : 8), "a panel holds two column groups, or one if there is one");
  const bool bad_sum = (l_run == 0.f) || (l_run != l_run);
  const float inv = bad_sum ? 1.f : (1.f / l_run) * a.rp_keep;
  auto out = [&](int row, int column) -> uint16_t* {
    return reinterpret_cast<uint16_t*>(a.o) + static_cast<int64_t>(q_start + row) * a.o_row_stride +
           static_cast<int64_t>(h) * a.o_head_stride + column;
  };
  // Whole rows by TMA (by the LSU before: 64 x 12 x 512, d = 64, 104.4 us, now 102.4; d = 128: 32 x 12 x 300 causal 51.2 -> 49.2,
  // 32 x 12 x 512 84 -> 81, 4 x 32 x 3000 causal 342 -> 335).  The warp that holds the sequence's end stores its rows itself: those
  // behind it are the next sequence's.
  const bool whole = ig + 32 <= sq;
  auto send = [&](int p) {
    if (whole) {
      if (lane == 0 && c0 * 32 + p * 64 < a.head_dim) {
        tma_store_3d(tm_o, smem_u32(piece) + (REUSE ? 0 : p * 4096), c0 * 32 + p * 64, q_start + ig, h);
        bulk_commit();
      }
    } else {
      stage_copy_out<CH>(piece + (REUSE ? 0 : p * 4096), out(ig, c0 * 32 + p * 64), a.o_row_stride, sq - ig,
                         a.head_dim / 8 - c0 * 4 - p * 8, lane);
    }
  };
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    uint32_t orr[32];
    if (have_acc) {
      tmem_ld32(tO + (c0 + i) * 32, orr);
      tmem_wait_ld();
    } else {
#pragma unroll
      for (int k = 0; k < 32; ++k) orr[k] = 0u;
    }
    if (STAGED && REUSE && i % 2 == 0) {
      if (lane == 0) bulk_wait_read();
      __syncwarp();
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        w[k] = pack_lowp<BF16>(__uint_as_float(orr[8 * v + 2 * k]) * inv, __uint_as_float(orr[8 * v + 2 * k + 1]) * inv);
      if constexpr (STAGED)
        *reinterpret_cast<uint4*>(piece + (REUSE ? 0 : i / 2) * 4096 + stage_offset<CH>(lane, (i & 1) * 4 + v)) = make_uint4(w[0], w[1], w[2], w[3]);
      else if (ok && ig + lane < sq && (c0 + i) * 32 + v * 8 < a.head_dim)
        *reinterpret_cast<uint4*>(out(ig + lane, (c0 + i) * 32 + v * 8)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if constexpr (STAGED && REUSE) {
      if (i % 2 == 1 || i + 1 == NC) {
        fence_async_smem();
        __syncwarp();
        if (ok) send(i / 2);
      }
    }
  }
  if constexpr (STAGED && !REUSE) {
    fence_async_smem();
    __syncwarp();
  }
  if (!ok) return;
  if (ig + lane < sq && c0 == 0) {
    const float lse = bad_sum ? -INFINITY : (m_run * a.scale + __logf(l_run));
    a.lse[(static_cast<int64_t>(b) * a.heads + h) * a.lse_stride + ig + lane] = lse;
  }
  if constexpr (STAGED && !REUSE) {
#pragma unroll
    for (int p = 0; p < (NC + 1) / 2; ++p) send(p);
    if (lane == 0 && whole) bulk_wait_read();
  }
}

// Padded batches.  A V tile that reaches behind its sequence's last token holds whatever the padding holds, and its
// probabilities there are zero: the rows are cleared, so that an infinity or a NaN in the padding stays out of the sum.
// One warp, behind the tile's load and ahead of the product.
template <int PANELS>
__device__ __forceinline__ void clear_v_rows(uint8_t* tile, int first, int lane) {
#pragma unroll
  for (int p = 0; p < PANELS; ++p)
    for (int i = first * 8 + lane; i < kBlockN * 8; i += 32)
      *reinterpret_cast<uint4*>(tile + p * 16384 + i * 16) = make_uint4(0, 0, 0, 0);
  fence_async_smem();
  __syncwarp();
}

// Rows [r0, r1) of sequence b's padded rows that hold no token (`first`, `len`: its run) get zeros, by `threads` threads.
__device__ __forceinline__ void zero_padding(const KernelArgs& a, int b, int h, int r0, int r1, int first, int len, int thread,
                                             int threads) {
  const int chunks = a.head_dim / 8;
  uint16_t* o = reinterpret_cast<uint16_t*>(a.o) + static_cast<int64_t>(b) * a.pad_rows * a.o_row_stride +
                static_cast<int64_t>(h) * a.o_head_stride;
  for (int i = r0 * chunks + thread; i < min(r1, a.pad_rows) * chunks; i += threads) {
    const int r = i / chunks;
    if (r < first || r >= first + len)
      *reinterpret_cast<uint4*>(o + r * a.o_row_stride + (i - r * chunks) * 8) = make_uint4(0, 0, 0, 0);
  }
}

// PADDED: see KernelArgs::pad_rows
template <int D, bool BF16, bool CAUSAL, bool DROPOUT, bool BLOCKSPARSE, int G, bool ROWS, Order ORDER, bool PADDED>
__global__ void __launch_bounds__(FwdCfg<D, G, ROWS>::kThreads, G == 1 ? 2 : 1)
fa_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
              const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o, const KernelArgs a) {
  constexpr bool TAKE = ORDER == kTake, LINEAR = ORDER != kPlain;
  using Cfg = FwdCfg<D, G, ROWS, TAKE>;
  // d = 128: P is handed over in two parts, so that P*V of the first 96 keys (64 in quads) runs while the rest is exponentiated; S of
  // the next tile waits for P*V there, and so tells that it is over.  Quads, us, whole and waited for -> now: 4 x 12 x 4096 causal with
  // dropout 298 -> 290, 2 x 16384 and 126 x 64, 4 heads 1486 -> 1450, causal 922 -> 892, 16 x 256 queries, 4096 keys 198 -> 190.
  constexpr bool kHalfP = !Cfg::kSeparateP;
  constexpr int kFirstSteps = kHalfP ? (Cfg::kRows ? 6 : 4) : 0;  // of 16 keys, in the first part
  extern __shared__ uint8_t smem_raw[];
  __shared__ FwdShared<ROWS ? 1 : TAKE ? 2 * G : G> sh;
  // block-sparse: key tiles this CTA visits (ascending), built from the layout table
  __shared__ uint16_t tile_list[BLOCKSPARSE ? kMaxSparseTiles : 1];
  __shared__ uint32_t tile_bits[BLOCKSPARSE ? kMaxSparseTiles / 32 : 1];

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // known to be the same in all lanes
  const int lane = tid & 31;

  auto decode = [&](uint32_t block) -> FwdBlock {
    FwdBlock x;
    if constexpr (LINEAR) tail_block(a, block, x.mp, x.h, x.b);
    else { x.b = blockIdx.z; x.h = blockIdx.y; x.mp = CAUSAL ? gridDim.x - 1 - blockIdx.x : blockIdx.x; }  // heavy tiles first
    x.q_start = a.cu_seqlens_q[PADDED ? 2 * x.b : x.b];
    x.sq = a.cu_seqlens_q[PADDED ? 2 * x.b + 1 : x.b + 1] - x.q_start;
    x.k_start = PADDED ? x.q_start : a.cu_seqlens_k[x.b];
    x.sk = PADDED ? x.sq : a.cu_seqlens_k[x.b + 1] - x.k_start;
    if constexpr (LINEAR && CAUSAL) {
      const int mp = (x.sq + G * kBlockM - 1) / (G * kBlockM) - 1 - x.mp;  // of the sequence's own tiles; empty blocks last
      if (!PADDED || mp >= 0) x.mp = mp;
    }
    return x;
  };
  auto without_queries = [&](const FwdBlock& x) -> bool { return LINEAR && CAUSAL && !PADDED ? x.mp < 0 : x.mp * G * kBlockM >= x.sq; };
  auto count_tiles = [&](FwdBlock& x) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int m0 = (x.mp * G + g) * kBlockM;
      int n = (x.sk + kBlockN - 1) / kBlockN;
      if (CAUSAL) n = min(n, m0 / kBlockN + 1);
      (g == 0 ? x.n0 : x.n1) = m0 < x.sq ? n : 0;
    }
    if (G == 1) x.n1 = 0;
  };
  FwdBlock first = decode(blockIdx.x);
  if constexpr (PADDED) {
    if (first.q_start < 0) return;
    if (without_queries(first))
      zero_padding(a, first.b, first.h, first.mp * G * kBlockM, (first.mp + 1) * G * kBlockM, first.q_start - first.b * a.pad_rows, first.sq,
                   tid, Cfg::kThreads);
  }
  // On the lengths alone: a grid announced with a long sequence consists mostly of blocks without queries, and everything ahead of
  // this line is their time.  With the status word and the barriers ahead of it too, which saves the others 0.1 us, us of an SM for such a
  // block 0.93-1.0 (d = 64), now 0.67-0.73; 0.47-0.58 (d = 128), now 0.39-0.48.  1 x 4096 and 63 x 128, 12 heads, d = 64: 232 -> 183 us.
  if (without_queries(first)) return;
  count_tiles(first);
  if (warp == Cfg::kSoftmaxWarps) {
    if (lane == 0) {
      sh.abort_flag = 0;
      if (TAKE) sh.blk[0] = first;
    }
    // a lane per barrier (those of a group from s_free on); taking over, with more barriers than lanes, a loop, which cost the others 0.5 %
    if (!TAKE && lane < kBarriers) mbar_init(smem_u32(&sh.q_full[0]) + lane * 8, lane >= 16 && lane < 22 ? Cfg::kArrivals : 1);
    for (int i = lane; i < (TAKE ? kTakeBarriers : 0); i += 32) {
      const uint64_t* bar = &sh.q_full[0] + i;
      const uint32_t count = bar >= &sh.s_free[0] && bar < &sh.o_full[0] ? Cfg::kArrivals
                             : bar >= &sh.blk_done[0] && bar < &sh.out_free ? Cfg::kSoftmaxWarps + 1 + (Cfg::kSeparateP ? 1 : 0) + (PADDED ? 1 : 0)  // all but the producer
                             : bar == &sh.out_free ? Cfg::kSoftmaxWarps
                             : bar >= &sh.stats_full[0] ? Cfg::kGroupWarps : 1;
      mbar_init(smem_u32(bar), count);
    }
    fence_mbar_init();
    fence_async_smem();
    __syncwarp();
  }

  if constexpr (BLOCKSPARSE) {
    // A key tile is visited when any 16-row block of this CTA's 128 * G query rows has its 256-column
    // key block in the layout; rows whose block is absent are masked inside the tile.  A ballot for 32 tiles, and places by counting
    // bits: one thread that went through flags for the CTA took about 1000 clk for 32 of them.  us, 4 x 16 x 4096, d = 64, 10, 25 and 100 %
    // of the blocks 116 -> 109, 158 -> 151, 376 -> 366, with dropout 162 -> 152, 236 -> 224, 623 -> 592.
    constexpr int kWarps = Cfg::kThreads / 32;
    const int mp = first.mp, b = first.b;
    const int n_kv = min((first.sk + kBlockN - 1) / kBlockN, kMaxSparseTiles);
    const int rb0 = mp * (G * kBlockM / 16), rb1 = min(a.bs_rows16, (first.sq + 15) >> 4);
    for (int c = warp; c * 32 < n_kv; c += kWarps) {
      const int j = c * 32 + lane;
      const int32_t* row = a.bs_iter + (static_cast<int64_t>(b) * a.bs_kblocks + (j >> 1)) * a.bs_rows16;
      int most = -1;  // (all loads at once: none decides about the next)
      // (causal: a key tile that starts behind the CTA's last query row is masked entirely)
      if (j < n_kv && rb0 < rb1 && !(CAUSAL && j * kBlockN > mp * G * kBlockM + G * kBlockM - 1))
#pragma unroll
        for (int i = 0; i < G * kBlockM / 16; ++i) most = max(most, row[min(rb0 + i, rb1 - 1)]);
      const uint32_t bits = __ballot_sync(0xffffffffu, most >= 0);
      if (lane == 0) tile_bits[c] = bits;
    }
    __syncthreads();
    int total = 0, upto[G] = {};  // listed key tiles; those up to the one that holds a query tile's diagonal
    for (int c = 0; c * 32 < n_kv; ++c) {
      const uint32_t bits = tile_bits[c];
      if (c % kWarps == warp && (bits >> lane & 1))
        tile_list[total + __popc(bits & ((1u << lane) - 1))] = static_cast<uint16_t>(c * 32 + lane);
      total += __popc(bits);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const int last = mp * G + g - c * 32;
        if (last >= 0) upto[g] += __popc(last >= 31 ? bits : bits & ((2u << last) - 1));
      }
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < G; ++g)
      (g == 0 ? first.n0 : first.n1) = (mp * G + g) * kBlockM < first.sq ? (CAUSAL ? upto[g] : total) : 0;
  }
  auto kv_tile = [&](int j) -> int {
    if constexpr (BLOCKSPARSE) return tile_list[j];
    else return j;
  };

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const uint32_t smem_q = smem_u32(smem);
  const uint32_t smem_k = smem_q + G * Cfg::kTileBytes;
  const uint32_t smem_v = smem_k + Cfg::kStages * Cfg::kTileBytes;
  const uint32_t smem_out = smem_v + Cfg::kStages * Cfg::kTileBytes;
  // the 128 rows from `row` on of one operand (one thread)
  auto load_tile = [&](uint32_t dst, const CUtensorMap* map, uint64_t& bar, int row, int h) {
    mbar_expect_tx(smem_u32(&bar), Cfg::kTileBytes);
    for (int p = 0; p < Cfg::kPanels; ++p) tma_load_3d(dst + p * 16384, map, smem_u32(&bar), p * 64, row, h);
  };
  auto load_q = [&](const FwdBlock& x, int g) {
    load_tile(smem_q + g * Cfg::kTileBytes, &tm_q, sh.q_full[g], x.q_start + (x.mp * G + g) * kBlockM, x.h);
  };

  // The producer asks for Q and the first K and V at once, ahead of everything else a CTA does: behind
  // the tensor memory, the register split and the barrier of the CTA the first load left 3100 clk after the start of a CTA and
  // the first scores came at 5600 (16 x 12 x 1000 causal, d = 128, 51 000 clk for eight key tiles).  With K waited for where it
  // is used (issuer) and the rows stored through shared memory (store_rows, 3500 clk before), us, before -> now: 16 x 12 x 1000
  // causal (d = 128) 97 -> 83; d = 64: 64 x 12 x 512 100 -> 95, 16 x 12 x 1024 87 -> 80, 8 x 12 x 4096 479 -> 465, 2 x 4 x 16384
  // causal 310 -> 307.
  const int first_max = max(first.n(0), first.n(G - 1));
  if (tid == 32 * Cfg::kSoftmaxWarps && first_max > 0) {
    for (int g = 0; g < G; ++g)
      if (first.n(g) > 0) load_q(first, g);
    load_tile(smem_k, &tm_k, sh.k_full[0], first.k_start + kv_tile(0) * kBlockN, first.h);
    load_tile(smem_v, &tm_v, sh.v_full[0], first.k_start + kv_tile(0) * kBlockN, first.h);
  }
  // Fail fast: once a CTA of this launch has abandoned a wait, those that start after it do not go on.  Quads look here and leave behind
  // the barrier, with their first loads ended.  In rows and padded batches, whose shorter walks would wait for the word, the idle warp
  // looks, and the CTA leaves at its first waits: 64 x 12 x 512 padded 94.8 -> 93.7 us, 8 heads of 100 tokens in a graph 5.13 -> 4.95 (in quads the same made
  // 4 x 12 x 4096, d = 128 with dropout, 539 -> 550).
  constexpr bool kLateLook = Cfg::kRows || PADDED;
  auto launch_failed = [&]() -> bool { return a.status && *reinterpret_cast<volatile int32_t*>(a.status) == a.launch_id; };
  if (warp == Cfg::kSoftmaxWarps + 1) {
    const bool failed = !kLateLook && lane == 0 && launch_failed();
    __syncwarp();
    tmem_alloc(smem_u32(&sh.tmem_base), Cfg::kTmemCols);
    if (lane == 0) sh.stop = failed;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem_base;
  if (!kLateLook && sh.stop) {
    if (tid == 32 * Cfg::kSoftmaxWarps && first_max > 0) {
      for (int g = 0; g < G; ++g)
        if (first.n(g) > 0) mbar_drain(smem_u32(&sh.q_full[g]), 0);
      mbar_drain(smem_u32(&sh.k_full[0]), 0);
      mbar_drain(smem_u32(&sh.v_full[0]), 0);
    }
    if (warp == Cfg::kSoftmaxWarps + 1) tmem_dealloc(tmem, Cfg::kTmemCols);
    return;
  }
  volatile int* abort_flag = &sh.abort_flag;

  // Block k of this CTA.  The softmax warps read it where they use it, to hold few registers across the tiles.
  auto block_at = [&](uint32_t k) -> std::conditional_t<TAKE, const FwdBlock&, FwdBlock> {
    if constexpr (TAKE) return sh.blk[k & 1];
    else return first;
  };
  // A warp has finished block k: waits for the next one, if any (or until a wait is abandoned).
  // idle: a softmax group without rows has no part in the block, which the others may be at for any time.
  auto next_block = [&](uint32_t k, bool idle = false) -> bool {
    if constexpr (!TAKE) return false;
    __syncwarp();
    if (elect_one()) mbar_arrive(smem_u32(&sh.blk_done[k & 1]));
    if (G == 2 && idle) mbar_wait_alive(smem_u32(&sh.blk_full[(k + 1) & 1]), (k >> 1) & 1, abort_flag, &sh.alive);
    return mbar_wait_warp<true>(smem_u32(&sh.blk_full[(k + 1) & 1]), (k >> 1) & 1, abort_flag) && sh.blk[(k + 1) & 1].mp >= 0;
  };

  // Causal calls with dropout in single tiles (quads) spilled 20-80 bytes with 96 and 48 registers; the four other warps do with 32 (104 x 256
  // + 32 x 128 = 80 x 384, what the CTA is launched with).  us: block-sparse, 25 % of the
  // blocks, 4 x 16 x 4096 151.6 -> 145.2, 16 x 12 x 2048 ragged 138.8 -> 130.1; dense 16 x 12 x 1000 86.1 -> 84.1, 4 x 12 x 4096 243.4 -> 239.2,
  // d = 128 100.7 -> 99.2 and 298.0 -> 296.8.
  // Without a causal mask the same made them 1-2.5 % slower (4 x 12 x 4096 442 -> 449, d = 128 544 -> 555).
  constexpr bool kMoreRegs = CAUSAL && DROPOUT && G == 1;
  if (warp >= Cfg::kSoftmaxWarps) reg_dealloc<kMoreRegs ? 32 : Cfg::kOtherRegs>();
  if (warp == Cfg::kSoftmaxWarps) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      bool ok = true;
      int loads_k = 0, loads_v = 0, loads_q[G] = {};  // so far
      uint32_t asked = 0;                             // requests so far
      // asked for with the loads of the last key tile: a block taken earlier would wait here while other SMs run dry
      auto take_next = [&]() {
        mbar_expect_tx(smem_u32(&sh.next_full), 16);
        clc_try_cancel(smem_u32(&sh.next), smem_u32(&sh.next_full));
        ++asked;
      };
      FwdBlock x = first;
      for (uint32_t k = 0; ok; ++k) {
        const int n_max = max(x.n(0), x.n(G - 1));
        for (int g = 0; g < G && ok; ++g) {
          if (x.n(g) == 0) continue;
          if (k > 0) {
            if (loads_q[g] > 0) ok = mbar_wait(smem_u32(&sh.q_empty[g]), (loads_q[g] & 1) ^ 1, abort_flag);
            if (!ok) break;
            load_q(x, g);
          }
          ++loads_q[g];
        }
        for (int j = 0; j < n_max && ok; ++j) {
          const int s = loads_k % Cfg::kStages;
          const uint32_t ph = ((loads_k / Cfg::kStages) & 1) ^ 1;
          const int row = x.k_start + kv_tile(j) * kBlockN;
          if (k > 0 || j > 0) {  // (the first ones are under way)
            if (loads_k >= Cfg::kStages) ok = mbar_wait(smem_u32(&sh.k_empty[s]), ph, abort_flag);
            if (!ok) break;
            load_tile(smem_k + s * Cfg::kTileBytes, &tm_k, sh.k_full[s], row, x.h);
          }
          ++loads_k;
          if (TAKE && G == 2) *const_cast<volatile uint32_t*>(&sh.alive) = loads_k;
          if (TAKE && j + 1 == n_max) take_next();
          if (k > 0 || j > 0) {
            if (loads_v >= Cfg::kStages) ok = mbar_wait(smem_u32(&sh.v_empty[s]), ph, abort_flag);
            if (ok && Cfg::kOutInV && j == 0) ok = mbar_wait(smem_u32(&sh.out_free), (k & 1) ^ 1, abort_flag);
            if (!ok) break;
            load_tile(smem_v + s * Cfg::kTileBytes, &tm_v, sh.v_full[s], row, x.h);
          }
          ++loads_v;
        }
        if (!TAKE || !ok) break;
        if (n_max == 0) take_next();
        // The next block with queries.  (Padded batches pass the others on too: their rows get zeros.  Else see kPassOnEvery.)
        bool more = false;
        while (true) {
          ok = mbar_wait(smem_u32(&sh.next_full), (asked - 1) & 1, abort_flag);
          if (!ok) break;
          uint32_t block;
          more = clc_answer(smem_u32(&sh.next), block);
          fence_async_smem();
          if (!more) break;
          more = !launch_failed();
          x = decode(block);
          if (!more || PADDED || !without_queries(x)) break;
          if (asked % kPassOnEvery == 0) {
            x.mp = x.sq = 0;
            break;
          }
          take_next();
        }
        if (!ok) break;
        if (!more) x.mp = -1;
        count_tiles(x);
        // its place is free once every role has finished block k - 1
        if (k >= 1) ok = mbar_wait(smem_u32(&sh.blk_done[(k + 1) & 1]), ((k - 1) >> 1) & 1, abort_flag);
        if (!ok) break;
        sh.blk[(k + 1) & 1] = x;
        mbar_arrive(smem_u32(&sh.blk_full[(k + 1) & 1]));
        if (!more) break;
      }
      for (int g = 0; g < G; ++g) mbar_drain_ring(&sh.q_full[g], 1, loads_q[g]);
      mbar_drain_ring(sh.k_full, Cfg::kStages, loads_k);
      mbar_drain_ring(sh.v_full, Cfg::kStages, loads_v);
      if (TAKE) mbar_drain_ring(&sh.next_full, 1, asked);
    }
  } else if (warp == Cfg::kSoftmaxWarps + 1) {
    // ------------------------------------------------------------------ MMA issuer
    // all 32 lanes run the loop, one elected lane issues (see mma_ss)
    constexpr uint32_t idesc_qk = make_idesc(BF16, false, false, kBlockM, kBlockN);
    constexpr uint32_t idesc_pv = make_idesc(BF16, false, true, kBlockM, D);
    const uint64_t desc_q = make_smem_desc(smem_q, 16, 1024);
    const uint64_t desc_k = make_smem_desc(smem_k, 16, 1024);
    const uint64_t desc_v = make_smem_desc(smem_v, 16384, 1024);
    // last: the block's last product of this group, which frees its Q
    auto issue_qk = [&](int g, int stage, bool last) {
      const uint64_t qa = desc_here(desc_at(desc_q, g * Cfg::kTileBytes));
      const uint64_t ka = desc_here(desc_at(desc_k, stage * Cfg::kTileBytes));
      const uint32_t tS = tmem + (g == 0 ? Cfg::kTmemS0 : Cfg::kTmemS1);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t off = (ks >> 2) * 16384 + (ks & 3) * 32;
          mma_ss(tS, desc_at(qa, off), desc_at(ka, off), idesc_qk, ks > 0);
        }
        mma_commit(smem_u32(&sh.s_full[g]));
        if (TAKE && last) mma_commit(smem_u32(&sh.q_empty[g]));
      }
    };
    // key steps [k0, k1) of 16; the last part reports the product, unless P comes in parts
    auto issue_pv = [&](int g, int stage, bool accumulate, int k0, int k1) {
      const uint64_t va = desc_here(desc_at(desc_v, stage * Cfg::kTileBytes));
      const uint32_t tO = tmem + (g == 0 ? Cfg::kTmemO0 : Cfg::kTmemO1);
      const uint32_t tP = tmem + (g == 0 ? Cfg::kTmemP0 : Cfg::kTmemP1);
      if (elect_one()) {
#pragma unroll
        for (int ks = k0; ks < k1; ++ks)
          mma_ts(tO, tP + ks * 8, desc_at(va, ks * 2048), idesc_pv, accumulate || ks > 0);
        if (!kHalfP && k1 == kBlockN / 16) mma_commit(smem_u32(&sh.o_full[g]));
      }
    };

    bool ok = true;
    int kv = 0, c[G] = {};         // key tiles of the blocks before; products of each group
    uint32_t k = 0, c_q[G] = {};   // block; blocks whose Q was loaded
    do {
      const FwdBlock x = block_at(k);
      int n_tiles[G];
      for (int g = 0; g < G; ++g) n_tiles[g] = __shfl_sync(0xffffffffu, x.n(g), 0);
      const int n_max = max(n_tiles[0], n_tiles[G - 1]);
      for (int g = 0; g < G; ++g)
        if (ok && n_tiles[g] > 0) ok = mbar_wait_warp<true>(smem_u32(&sh.q_full[g]), c_q[g]++ & 1, abort_flag);
      if constexpr (Cfg::kSeparateP) {
        // this warp issues only the score products; the next one issues P*V
        for (int j = 0; j < n_max && ok; ++j) {
          const int s = (kv + j) % Cfg::kStages;
          ok = mbar_wait_warp<true>(smem_u32(&sh.k_full[s]), ((kv + j) / Cfg::kStages) & 1, abort_flag);
#pragma unroll
          for (int g = 0; g < G; ++g) {
            if (ok && j < n_tiles[g]) {
              if (c[g] > 0) ok = mbar_wait_warp<true>(smem_u32(&sh.s_free[g]), (c[g] & 1) ^ 1, abort_flag);
              if (ok) {
                tc_fence_after();
                issue_qk(g, s, j + 1 == n_tiles[g]);
                ++c[g];
              }
            }
          }
          if (ok && elect_one()) mma_commit(smem_u32(&sh.k_empty[s]));
        }
      } else if (n_max > 0) {
        if (ok) ok = mbar_wait_warp<true>(smem_u32(&sh.k_full[kv % Cfg::kStages]), (kv / Cfg::kStages) & 1, abort_flag);
        if (ok) {
          tc_fence_after();
#pragma unroll
          for (int g = 0; g < G; ++g)
            if (n_tiles[g] > 0) issue_qk(g, kv % Cfg::kStages, n_tiles[g] == 1);
          if (elect_one()) mma_commit(smem_u32(&sh.k_empty[kv % Cfg::kStages]));
        }
        for (int j = 0; j < n_max && ok; ++j) {
          const int s = (kv + j) % Cfg::kStages;
          const int sn = (kv + j + 1) % Cfg::kStages;
          const bool has_next = j + 1 < n_max;
          auto wait_k = [&]() { ok = mbar_wait_warp<true>(smem_u32(&sh.k_full[sn]), ((kv + j + 1) / Cfg::kStages) & 1, abort_flag); };
          ok = mbar_wait_warp<true>(smem_u32(&sh.v_full[s]), ((kv + j) / Cfg::kStages) & 1, abort_flag);
          if (PADDED && ok && (j + 1) * kBlockN > x.sk)
            clear_v_rows<Cfg::kPanels>(smem + (smem_v - smem_q) + s * Cfg::kTileBytes, x.sk - j * kBlockN, lane);
          // K of the next tile is waited for behind P V of this one, which does not need it (its load takes about 2000 clk where
          // two CTAs with a stage each share an SM).  Pairs with dropout and without a causal mask wait ahead of it: their two groups
          // then take turns better (us: 2 x 16384 and 126 x 64 tokens, 4 heads 1603 -> 1486, 16 x 256 queries, 4096 keys, 16 heads
          // 209 -> 197; with a causal mask no difference).
          bool k_here = false;
          if (G == 2 && DROPOUT && !CAUSAL && ok && has_next) {
            wait_k();
            k_here = true;
          }
#pragma unroll
          for (int g = 0; g < G; ++g) {
            if (ok && j < n_tiles[g]) {
              const bool more = j + 1 < n_tiles[g];
              if constexpr (kHalfP) {
                ok = mbar_wait_warp<true>(smem_u32(&sh.p_half[g]), c[g] & 1, abort_flag);
                if (ok) {
                  tc_fence_after();
                  issue_pv(g, s, j > 0, 0, kFirstSteps);
                }
              }
              if (ok) ok = mbar_wait_warp<true>(smem_u32(&sh.p_full[g]), c[g] & 1, abort_flag);
              if (ok) {
                tc_fence_after();
                issue_pv(g, s, j > 0, kFirstSteps, kBlockN / 16);
                ++c[g];
                if (more) {
                  if (!k_here) wait_k();
                  k_here = true;
                  if (ok) issue_qk(g, sn, j + 2 == n_tiles[g]);
                } else if (kHalfP) {  // (S of the next tile reports the others)
                  if (elect_one()) mma_commit(smem_u32(&sh.o_full[g]));
                }
              }
            }
          }
          if (!ok) break;
          if (elect_one()) {
            mma_commit(smem_u32(&sh.v_empty[s]));
            if (has_next) mma_commit(smem_u32(&sh.k_empty[sn]));
          }
        }
      }
      kv += n_max;
    } while (ok && next_block(k++));
    mma_drain(smem_u32(&sh.drained[0]));
  } else if (warp == Cfg::kSoftmaxWarps + 2) {
    // ------------------------------------------------------------------ second MMA issuer (d = 64): P*V
    if constexpr (Cfg::kSeparateP) {
      constexpr uint32_t idesc_pv = make_idesc(BF16, false, true, kBlockM, D);
      const uint64_t desc_v = make_smem_desc(smem_v, 16384, 1024);
      bool ok = true;
      int kv = 0, c[G] = {};  // as above
      uint32_t k = 0;
      do {
        const FwdBlock x = block_at(k);
        int n_tiles[G];
        for (int g = 0; g < G; ++g) n_tiles[g] = __shfl_sync(0xffffffffu, x.n(g), 0);
        const int n_max = max(n_tiles[0], n_tiles[G - 1]);
        for (int j = 0; j < n_max && ok; ++j, ++kv) {
          const int s = kv % Cfg::kStages;
          ok = mbar_wait_warp<true>(smem_u32(&sh.v_full[s]), (kv / Cfg::kStages) & 1, abort_flag);
          if (!ok) break;
          if (PADDED && (j + 1) * kBlockN > x.sk)
            clear_v_rows<Cfg::kPanels>(smem + (smem_v - smem_q) + s * Cfg::kTileBytes, x.sk - j * kBlockN, lane);
          const uint64_t va = desc_here(desc_at(desc_v, s * Cfg::kTileBytes));
#pragma unroll
          for (int g = 0; g < G; ++g) {
            if (ok && j < n_tiles[g]) {
              ok = mbar_wait_warp<true>(smem_u32(&sh.p_full[g]), c[g] & 1, abort_flag);
              if (ok) {
                tc_fence_after();
                ++c[g];
                const uint32_t tO = tmem + (g == 0 ? Cfg::kTmemO0 : Cfg::kTmemO1);
                const uint32_t tP = tmem + (g == 0 ? Cfg::kTmemP0 : Cfg::kTmemP1);
                if (elect_one()) {
#pragma unroll
                  for (int ks = 0; ks < kBlockN / 16; ++ks)
                    mma_ts(tO, tP + ks * 8, desc_at(va, ks * 2048), idesc_pv, j > 0 || ks > 0);
                  mma_commit(smem_u32(&sh.o_full[g]));
                }
              }
            }
          }
          if (!ok) break;
          if (elect_one()) mma_commit(smem_u32(&sh.v_empty[s]));
        }
      } while (ok && next_block(k++));
      mma_drain(smem_u32(&sh.drained[1]));
    }
  } else if (kLateLook && warp == Cfg::kSoftmaxWarps + 3) {
    if (lane == 0 && launch_failed()) *abort_flag = 1;
    if constexpr (PADDED) {
      uint32_t k = 0;
      do {
        const FwdBlock x = block_at(k);
        zero_padding(a, x.b, x.h, x.mp * G * kBlockM, (x.mp + 1) * G * kBlockM, x.q_start - x.b * a.pad_rows, x.sq, lane, 32);
      } while (next_block(k++));
    }
  } else if (Cfg::kRows && warp < Cfg::kSoftmaxWarps) {
    // ------------------------------------------------------------------ softmax groups, one thread per query row
    reg_alloc<Cfg::kSoftmaxRegs>();
    const int g = (G == 1) ? 0 : warp >> 2;
    const int row = tid & 127;
    const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + (g == 0 ? Cfg::kTmemS0 : Cfg::kTmemS1) + lane_sel;
    const uint32_t tO = tmem + (g == 0 ? Cfg::kTmemO0 : Cfg::kTmemO1) + lane_sel;
    const uint32_t tP = tmem + (g == 0 ? Cfg::kTmemP0 : Cfg::kTmemP1) + lane_sel;
    bool ok = true, s_early = false;
    const uint64_t c2 = pack_f2(a.scale_log2, a.scale_log2);
    int t = 0, n;             // key tiles so far, of the block
    uint32_t k = 0, c_o = 0;  // block; blocks with key tiles before
    do {
    const FwdBlock& x = block_at(k);
    n = x.n(g);
    float m_run = -INFINITY, l_run = 0.f;
    const int free_tiles = CAUSAL ? min(x.sk / kBlockN, x.mp * G + g) : x.sk / kBlockN;  // key tiles without a mask

    for (int j = 0; j < n && ok; ++j, ++t) {
      const int col0 = kv_tile(j) * kBlockN;
      int32_t bs_it = 0;
      if constexpr (BLOCKSPARSE) {
        const int b = x.b, ig = (x.mp * G + g) * kBlockM + row;
        bs_it = (ig >> 4) < a.bs_rows16
                    ? a.bs_iter[(static_cast<int64_t>(b) * a.bs_kblocks + (col0 >> 8)) * a.bs_rows16 + (ig >> 4)]
                    : -1;
      }
      if (!Cfg::kSeparateP || !__all_sync(0xffffffffu, s_early)) ok = mbar_wait_warp<!Cfg::kSeparateP>(smem_u32(&sh.s_full[g]), t & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      uint32_t sr[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, sr[c]);
      tmem_wait_ld();
      if constexpr (Cfg::kSeparateP) {
        tc_fence_before();
        mbar_arrive(smem_u32(&sh.s_free[g]));
      }

      if (kv_tile(j) >= free_tiles) {
        const int ig = (x.mp * G + g) * kBlockM + row, sk = x.sk;  // query index within the sequence
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int col = col0 + c * 32 + i;
            bool valid = col < sk;
            if (CAUSAL) valid = valid && (col <= ig);
            if (!valid) sr[c][i] = __float_as_uint(-INFINITY);
          }
      }
      if constexpr (BLOCKSPARSE) {
        // a 16-row block that is not in the layout for this 256-column key block sees -inf
        if (bs_it < 0) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) sr[c][i] = __float_as_uint(-INFINITY);
        }
      }

      float mxa = -INFINITY, mxb = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          mxa = max3(mxa, __uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1]));
          mxb = max3(mxb, __uint_as_float(sr[c][i + 2]), __uint_as_float(sr[c][i + 3]));
        }
      const float m_new = max3(m_run, mxa, mxb);

      // The running max is only raised when it would grow by more than 2^8 in the exponent:
      // until then the stale max keeps every p below 256 and saves rescaling O.
      const bool grow = (m_new - m_run) * a.scale_log2 > 8.f;
      const float m_next = grow ? m_new : m_run;
      const float alpha = (!grow || m_run == -INFINITY) ? (grow ? 0.f : 1.f) : ex2f((m_run - m_new) * a.scale_log2);
      m_run = m_next;
      const float mc = (m_next == -INFINITY) ? 0.f : m_next * a.scale_log2;
      const uint64_t nmc2 = pack_f2(-mc, -mc);

      // p = exp2(s * c - m * c): packed fma, one ex2 per element, packed row sum, 16-bit pack
      uint32_t pk[64];
      uint64_t sum_a = 0ull, sum_b = 0ull;
      auto expo = [&](int from, int to) {
#pragma unroll
        for (int e = from; e < to; e += 4) {
          const int c = e / 32, i = e % 32;
          float p0, p1, p2, p3;
          unpack_f2(fma2(pack_f2(__uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1])), c2, nmc2), p0, p1);
          unpack_f2(fma2(pack_f2(__uint_as_float(sr[c][i + 2]), __uint_as_float(sr[c][i + 3])), c2, nmc2), p2, p3);
          p0 = ex2f(p0); p1 = ex2f(p1); p2 = ex2f(p2); p3 = ex2f(p3);
          const uint64_t p01 = pack_f2(p0, p1), p23 = pack_f2(p2, p3);
          sum_a = add2(sum_a, p01);
          sum_b = add2(sum_b, p23);
          pk[c * 16 + i / 2] = pack_lowp<BF16>(p0, p1);
          pk[c * 16 + i / 2 + 1] = pack_lowp<BF16>(p2, p3);
        }
      };
      // P V of the tile before, and S of the next tile (below), are over by the time they are needed, as a rule: looked for where nothing
      // waits for the answer, which takes 200 clk beside the other CTA's exponentials.  us: 64 x 12 x 512 83.5 -> 82.6, ragged
      // batches of 12 heads up to 256 tokens 71.7 -> 70.8, 512 90.1 -> 88.6 (quads, four warps to a scheduler: no change or slower).
      const bool o_early = Cfg::kSeparateP && j > 0 && mbar_test(smem_u32(&sh.o_full[g]), (t & 1) ^ 1);
      expo(0, 64);
      // P*V of the previous tile must have finished before O is rescaled or its P buffer reused.  With P over S (d = 128) it has: these
      // scores were issued behind it.  (Else: half of the exponentials are still to come, and by now it has, as a rule.)
      if (j > 0) {
        if constexpr (Cfg::kSeparateP) {
          if (!__all_sync(0xffffffffu, o_early)) ok = mbar_wait_warp(smem_u32(&sh.o_full[g]), (t & 1) ^ 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
        }
        if (__any_sync(0xffffffffu, grow)) {
          const uint64_t alpha2 = pack_f2(alpha, alpha);
#pragma unroll
          for (int c = 0; c < D / 16; ++c) {
            uint32_t orr[16];
            tmem_ld16(tO + c * 16, orr);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              float lo, hi;
              unpack_f2(mul2(pack_f2(__uint_as_float(orr[i]), __uint_as_float(orr[i + 1])), alpha2), lo, hi);
              orr[i] = __float_as_uint(lo);
              orr[i + 1] = __float_as_uint(hi);
            }
            tmem_st16(tO + c * 16, orr);
          }
        }
      }
      // Hand P to the tensor core through tensor memory.  In parts: three quarters first, and reported behind the next eight
      // exponentials, when the stores have been taken.  us, halves that are reported at once and a wait for P V ahead of the first -> no
      // wait -> now: 4 x 12 x 4096 354 -> 342 -> 342, 4 x 12 x 8192 causal 660 -> 639 -> 637, 16 x 12 x 1000 120 -> 117 -> 115, 64 x 12 x
      // 300 92.3 -> 91.0 -> 90.5.  (Traces, 4 x 12 x 4096: a group's 3560 clk a tile are 200 for the scores, 300 for the maximum, 1500
      // exponentials beside the other group's, 170 of that wait, 1070 from P to the next S.)
      tmem_st32(tP, reinterpret_cast<uint32_t(&)[32]>(pk[0]));
      if constexpr (kHalfP) {
        static_assert(!Cfg::kRows || kFirstSteps == 6, "96 keys");
        expo(64, 96);
        tmem_st16(tP + 32, reinterpret_cast<uint32_t(&)[16]>(pk[32]));
        expo(96, 104);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(smem_u32(&sh.p_half[g]));
        expo(104, 128);
      } else {
        expo(64, 96);
        s_early = mbar_test(smem_u32(&sh.s_full[g]), (t & 1) ^ 1);
        expo(96, 128);
      }
      {
        float s0, s1;
        unpack_f2(add2(sum_a, sum_b), s0, s1);
        l_run = l_run * alpha + (s0 + s1);
      }
      if constexpr (kHalfP) tmem_st16(tP + 48, reinterpret_cast<uint32_t(&)[16]>(pk[48]));
      else tmem_st32(tP + 32, reinterpret_cast<uint32_t(&)[32]>(pk[32]));
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(smem_u32(&sh.p_full[g]));
    }

    // ---------------- epilogue: O = acc / (sum * p_keep), LSE
    const int m_first = (x.mp * G + g) * kBlockM, sq = x.sq;
    if (m_first < sq) {
      if (n > 0 && ok) {
        ok = mbar_wait_warp<true>(smem_u32(&sh.o_full[g]), (kHalfP ? c_o : t - 1) & 1, abort_flag);
        tc_fence_after();
      }
      // (every product that reads this group's Q has finished: without other blocks its tile takes the output)
      store_rows<BF16, D / 32, Cfg::kBoxRows, TAKE && !Cfg::kOutInV>(a, &tm_o, tO, 0, n > 0 && ok, ok, m_first + (warp & 3) * 32, lane, sq, x.q_start, x.b, x.h,
                               m_run, l_run, TAKE ? smem + ((Cfg::kOutInV ? smem_v : smem_out) - smem_q) + warp * Cfg::kOutPiece
                                                  : smem + g * Cfg::kTileBytes + (warp & 3) * (D * 64));
    }
    if (n > 0) ++c_o;
    if constexpr (Cfg::kOutInV) {
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh.out_free));
    }
    } while (ok && next_block(k++, n == 0));
    if (TAKE && lane == 0) bulk_wait_read();
  } else if (warp < Cfg::kSoftmaxWarps) {
    // ------------------------------------------------------------------ softmax warps
    // A warp owns 16 query rows.  It reads their scores with the 16x256b shape, in which a thread holds rows r8 and
    // r8 + 8 and, of every 8-column unit, two adjacent columns: the ownership pattern of the reference's mask
    // generator (one Philox call covers exactly one thread's part of a 16 x 16 patch, QuadPhilox).
    reg_alloc<kMoreRegs ? 104 : Cfg::kSoftmaxRegs>();
    const int g = (G == 1) ? 0 : warp >> 3;
    const int hh = (warp >> 2) & 1, wq = warp & 3;
    const int r8 = lane >> 2, q4 = lane & 3;
    const uint32_t lane_sel = static_cast<uint32_t>(wq * 32 + hh * 16) << 16;
    const uint32_t tS = tmem + (g == 0 ? Cfg::kTmemS0 : Cfg::kTmemS1) + lane_sel;
    const uint32_t tO = tmem + (g == 0 ? Cfg::kTmemO0 : Cfg::kTmemO1) + lane_sel;
    const uint32_t tP = tmem + (g == 0 ? Cfg::kTmemP0 : Cfg::kTmemP1) + lane_sel;
    bool ok = true;
    const uint64_t c2 = pack_f2(a.scale_log2, a.scale_log2);
    int t = 0, n;             // key tiles so far, of the block
    uint32_t k = 0, c_o = 0, c_s = 0;  // block; blocks with key tiles before, with queries before
    do {
    const FwdBlock& x = block_at(k);
    n = x.n(g);
    // rows r8 (u = 0) and r8 + 8 (u = 1); l_run: this thread's share of the row sum (its 32 columns per tile)
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    const int free_tiles = CAUSAL ? min(x.sk / kBlockN, x.mp * G + g) : x.sk / kBlockN;  // key tiles without a mask

    const int64_t bh_sub =
        (static_cast<int64_t>(x.b) * a.drop.heads_total + a.drop.head_offset + x.h) * 256;
    QuadPhilox<8> qp;
    float thr_term = 0.f;
    if constexpr (DROPOUT) {
      qp.init(a.drop, bh_sub, lane);
      thr_term = fa_keep_thr_term(a.drop.threshold);
    }
    auto arrive_warp = [&](uint64_t& bar) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar));
    };

    for (int j = 0; j < n && ok; ++j, ++t) {
      const int col0 = kv_tile(j) * kBlockN;
      int32_t bs_it = 0;
      if constexpr (BLOCKSPARSE) {
        const int i16 = ((x.mp * G + g) * kBlockM + wq * 32 + hh * 16) >> 4;
        bs_it = i16 < a.bs_rows16
                    ? a.bs_iter[(static_cast<int64_t>(x.b) * a.bs_kblocks + (col0 >> 8)) * a.bs_rows16 + i16]
                    : -1;
      }
      // (us, by columns -> by tiles: 8 heads x 3000 causal 35.7 -> 35.5, 2 x 12 x 8192 causal with dropout at d = 128 516 -> 501; single tiles
      // without a causal mask 2-3 % slower)
      const bool need_mask = TAKE || (!BLOCKSPARSE && (CAUSAL || G == 2)) ? j >= free_tiles
                                  : (col0 + kBlockN > x.sk) || (CAUSAL && (col0 + kBlockN - 1 > (x.mp * G + g) * kBlockM)) ||
                                        (BLOCKSPARSE && bs_it < 0);
      // -inf for columns without a key, keys behind the diagonal and 16-row blocks that are not in the layout; s[]
      // holds the units from unit0 on, s[4 * unit + 2 * u + c] = (row r8 + 8 u, column 8 unit + 2 q4 + c)
      auto mask = [&](auto& s, int unit0) {
        constexpr int kValues = sizeof(s) / 4;
        const int sk = x.sk, row0 = (x.mp * G + g) * kBlockM + wq * 32 + hh * 16;  // of the warp; query index within the sequence
#pragma unroll
        for (int i = 0; i < kValues; ++i) {
          const int col = col0 + (unit0 + (i >> 2)) * 8 + 2 * q4 + (i & 1);
          bool valid = col < sk;
          if (CAUSAL) valid = valid && (col <= row0 + r8 + ((i >> 1) & 1) * 8);
          if (BLOCKSPARSE) valid = valid && bs_it >= 0;
          if (!valid) s[i] = __float_as_uint(-INFINITY);
        }
      };
      ok = mbar_wait_warp<true>(smem_u32(&sh.s_full[g]), t & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      uint32_t sr[64];
      tmem_ld_quad32(tS, reinterpret_cast<uint32_t(&)[32]>(sr[0]));
      tmem_ld_quad32(tS + 64, reinterpret_cast<uint32_t(&)[32]>(sr[32]));
      tmem_wait_ld();
      if constexpr (Cfg::kSeparateP && !DROPOUT) arrive_warp(sh.s_free[g]);
      if (need_mask) mask(sr, 0);

      // Row maxima.  The running max is only raised when it would grow by more than 2^8 in the exponent: until then
      // the stale max keeps every p below 256 and saves rescaling O.  Whether any row of the warp grows
      // shows without putting the quads' columns together.
      float mx[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float mxa = -INFINITY, mxb = -INFINITY;
#pragma unroll
        for (int unit = 0; unit < 16; unit += 2) {
          mxa = max3(mxa, __uint_as_float(sr[4 * unit + 2 * u]), __uint_as_float(sr[4 * unit + 2 * u + 1]));
          mxb = max3(mxb, __uint_as_float(sr[4 * unit + 4 + 2 * u]), __uint_as_float(sr[4 * unit + 5 + 2 * u]));
        }
        mx[u] = max3(m_run[u], mxa, mxb);
      }
      const bool grows = (mx[0] - m_run[0]) * a.scale_log2 > 8.f || (mx[1] - m_run[1]) * a.scale_log2 > 8.f;
      if (__any_sync(0xffffffffu, grows)) {
        float alpha[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          float m_new = fmaxf(mx[u], __shfl_xor_sync(0xffffffffu, mx[u], 1));
          m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 2));
          const bool grow = (m_new - m_run[u]) * a.scale_log2 > 8.f;
          alpha[u] = (!grow || m_run[u] == -INFINITY) ? (grow ? 0.f : 1.f)
                                                      : ex2f((m_run[u] - m_new) * a.scale_log2);
          if (grow) m_run[u] = m_new;
          l_run[u] *= alpha[u];
        }
        if (j > 0) {
          // P*V of the previous tile must have finished before O is rescaled (with P in parts: see the rows)
          if constexpr (!kHalfP) {
            ok = mbar_wait_warp<true>(smem_u32(&sh.o_full[g]), (t & 1) ^ 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
          }
          const uint64_t al[2] = {pack_f2(alpha[0], alpha[0]), pack_f2(alpha[1], alpha[1])};
#pragma unroll 1
          for (int col = 0; col < D; col += 32) {
            uint32_t orr[16];
            tmem_ld_quad16(tO + col, orr);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              float lo, hi;
              unpack_f2(mul2(pack_f2(__uint_as_float(orr[i]), __uint_as_float(orr[i + 1])), al[(i >> 1) & 1]), lo, hi);
              orr[i] = __float_as_uint(lo);
              orr[i + 1] = __float_as_uint(hi);
            }
            tmem_st_quad16(tO + col, orr);
          }
          tmem_wait_st();
        }
      }
      uint64_t nmc2[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float mc = (m_run[u] == -INFINITY) ? 0.f : m_run[u] * a.scale_log2;
        nmc2[u] = pack_f2(-mc, -mc);
      }

      // p = exp2(s * c - m * c): packed fma, one ex2 per element, packed row sum, 16-bit pack.  The row sum takes the
      // un-dropped p, P*V takes p times the keep factor (1 or 0).  64 columns after the other; s[] holds those of `half`.
      uint64_t sum_a[2] = {0ull, 0ull}, sum_b[2] = {0ull, 0ull};
      if constexpr (DROPOUT) {
        int64_t it_index;
        if constexpr (BLOCKSPARSE) it_index = bs_it;
        else it_index = fa_iter_index(CAUSAL, col0 >> a.drop.n_shift, ((x.mp * G + g) * kBlockM + wq * 32 + hh * 16) >> 4,
                                      (x.sq + 15) >> 4, a.drop.n_shift);
        qp.set_tile(a.drop, it_index, col0);
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t kw[DROPOUT ? 4 : 1][4];
        uint32_t sh_[DROPOUT ? 32 : 1];
        if constexpr (DROPOUT) {
          // The second half's scores are read again (the first pass was for the maxima): 32 instead of 64 of them live beside
          // the keep words of the half's four calls, kw[grp][2 * u + v] = row u, columns 16 grp + 8 v + 2 q4 (+1 high).  (With
          // the first half read again too, 8 x 12 x 4096 took 932 us instead of 906.)
          if (half == 1) tmem_ld_quad32(tS + 64, sh_);
#pragma unroll
          for (int grp = 0; grp < 4; ++grp) qp.start(half * 4 + grp, kw[grp]);
#pragma unroll
          for (int r = 2; r < 7; ++r)
#pragma unroll
            for (int k = 0; k < 4; ++k) QuadPhilox<8>::round(a.drop, kw[k], r);
          if (half == 1) {
            tmem_wait_ld();
            if (Cfg::kSeparateP) arrive_warp(sh.s_free[g]);
            if (need_mask) mask(sh_, 8);
          }
        }
        const uint32_t* s = DROPOUT && half == 1 ? sh_ : sr + half * 32;
        uint32_t pk[16];  // [2 * unit + u]: the 16x128b register of (row u, packed column pair 4 * unit + q4)
#pragma unroll
        for (int unit = 0; unit < 8; unit += 2) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            float p0, p1, p2, p3;
            unpack_f2(fma2(pack_f2(__uint_as_float(s[4 * unit + 2 * u]), __uint_as_float(s[4 * unit + 2 * u + 1])), c2, nmc2[u]), p0, p1);
            unpack_f2(fma2(pack_f2(__uint_as_float(s[4 * unit + 4 + 2 * u]), __uint_as_float(s[4 * unit + 5 + 2 * u])), c2, nmc2[u]), p2, p3);
            p0 = ex2f(p0); p1 = ex2f(p1); p2 = ex2f(p2); p3 = ex2f(p3);
            const uint64_t p01 = pack_f2(p0, p1), p23 = pack_f2(p2, p3);
            sum_a[u] = add2(sum_a[u], p01);
            sum_b[u] = add2(sum_b[u], p23);
            if constexpr (DROPOUT) {
              const uint32_t w01 = kw[unit / 2][2 * u], w23 = kw[unit / 2][2 * u + 1];
              unpack_f2(mul2(p01, pack_f2(fa_keep_factor_lo(w01, thr_term), fa_keep_factor_hi(w01, thr_term))), p0, p1);
              unpack_f2(mul2(p23, pack_f2(fa_keep_factor_lo(w23, thr_term), fa_keep_factor_hi(w23, thr_term))), p2, p3);
            }
            pk[2 * unit + u] = pack_lowp<BF16>(p0, p1);
            pk[2 * unit + 2 + u] = pack_lowp<BF16>(p2, p3);
          }
        }
        if (!kHalfP && half == 0 && j > 0) {
          // P*V of the previous tile must have finished before its P buffer is reused
          ok = mbar_wait_warp<true>(smem_u32(&sh.o_full[g]), (t & 1) ^ 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
        }
        // hand P to the tensor core through tensor memory
        tmem_st_pair16(tP + half * 32, pk);
        if (kHalfP && half == 0) {
          tmem_wait_st();
          arrive_warp(sh.p_half[g]);
        }
      }
      if (ok) {
        tmem_wait_st();
        arrive_warp(sh.p_full[g]);
      }
      if (!ok) break;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float s0, s1;
        unpack_f2(add2(sum_a[u], sum_b[u]), s0, s1);
        l_run[u] += s0 + s1;
      }
    }

    // ---------------- epilogue: O = acc / (sum * p_keep), LSE.  One thread per query row (32 rows per warp, half of the
    // columns): the statistics of a row pass through shared memory.
    const int m_first = (x.mp * G + g) * kBlockM;
    if (m_first < x.sq) {
      float2* stats = sh.row_stats[TAKE ? 2 * g + (k & 1) : g];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float l = l_run[u];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        if (q4 == 0) stats[wq * 32 + hh * 16 + u * 8 + r8] = make_float2(m_run[u], l);
      }
      if constexpr (TAKE) {
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sh.stats_full[g]));
        if (ok) ok = mbar_wait_warp<true>(smem_u32(&sh.stats_full[g]), c_s++ & 1, abort_flag);
      } else {
        named_barrier_sync(1 + g, 32 * Cfg::kGroupWarps);  // every warp of the group comes here, also after an abandoned wait
      }
      if (n > 0 && ok) {
        ok = mbar_wait_warp<true>(smem_u32(&sh.o_full[g]), (kHalfP ? c_o : t - 1) & 1, abort_flag);
        tc_fence_after();
      }
      const float2 st = stats[wq * 32 + lane];
      uint8_t* piece = TAKE ? smem + (smem_out - smem_q) + warp * Cfg::kOutPiece : smem + g * Cfg::kTileBytes + (wq * 2 + hh) * (D * 32);
      store_rows<BF16, D / 64, Cfg::kBoxQuads, TAKE>(a, &tm_o, tO - (static_cast<uint32_t>(hh * 16) << 16), hh * (D / 64),
                               n > 0 && ok, ok, m_first + wq * 32, lane, x.sq, x.q_start, x.b, x.h, st.x, st.y, piece);
    }
    if (n > 0) ++c_o;
    } while (ok && next_block(k++, n == 0));
    if (TAKE && lane == 0) bulk_wait_read();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == Cfg::kSoftmaxWarps + 1) {
    tmem_dealloc(tmem, Cfg::kTmemCols);
    if (lane == 0 && sh.abort_flag && a.status) {
      atomicExch(a.status, a.launch_id);  // stops the CTAs of this launch that have not started yet
      atomicExch(a.status + 2, 1);  // sticky: read by the host
    }
  }
}

template <int D, bool BF16, bool CAUSAL, bool DROPOUT, bool BS, int G, bool ROWS, bool PADDED = false, Order ORDER = kPlain>
cudaError_t launch_groups(const FwdLaunch& l, cudaStream_t stream) {
  dim3 grid((l.max_seqlen_q + G * kBlockM - 1) / (G * kBlockM), l.args.heads, l.args.batch);
  // (padded batches take pairs at d = 64 only where all blocks start at once: no batch of theirs is uneven)
  if constexpr (ORDER == kPlain && !(PADDED && D == 64 && G == 2)) {
    const Order order = grid_order<D, CAUSAL, DROPOUT, BS, G, ROWS>(l);
    if constexpr (kCanTake<DROPOUT, BS>)
      if (order == kTake) return launch_groups<D, BF16, CAUSAL, DROPOUT, BS, G, ROWS, PADDED, kTake>(l, stream);
    // (in rows, pairs and padded batches beyond 512 tokens always take over: see take_over_pays)
    if constexpr (CAUSAL && !(kCanTake<DROPOUT, BS> && ROWS && (G == 2 || PADDED)))
      if (order == kLinear) return launch_groups<D, BF16, CAUSAL, DROPOUT, BS, G, ROWS, PADDED, kLinear>(l, stream);
  }
  auto kernel = fa_fwd_kernel<D, BF16, CAUSAL, DROPOUT, BS, G, ROWS, ORDER, PADDED>;
  using Cfg = FwdCfg<D, G, ROWS, ORDER == kTake>;
  static SmemLimitFlags smem_limit_set;  // one per template instantiation of this function
  cudaError_t e = set_smem_limit_once(kernel, Cfg::kSmemBytes, smem_limit_set);
  if (e != cudaSuccess) return e;
  KernelArgs args = l.args;
  if constexpr (ORDER != kPlain) {
    set_tail_grid(&args, grid.x, CAUSAL && tail_order(l) ? int64_t(4) * D * l.max_seqlen_k : 0);  // K and V
    grid = dim3(grid.x * grid.y * grid.z, 1, 1);
  }
  kernel<<<grid, Cfg::kThreads, Cfg::kSmemBytes, stream>>>(l.tm_q, l.tm_k, l.tm_v, l.tm_o, args);
  return cudaGetLastError();
}

template <int D, bool CAUSAL, bool DROPOUT>
int box_columns(const FwdLaunch& l) {
  if (rows_layout<D, DROPOUT>(l)) return FwdCfg<D, 1, true>::kBoxRows;  // (pairs too)
  return one_tile_per_cta<D, CAUSAL, DROPOUT>(l) ? FwdCfg<D, 1, false>::kBoxQuads : FwdCfg<D, 2, false>::kBoxQuads;
}

template <int D, bool BF16, bool CAUSAL, bool DROPOUT, bool BS, bool PADDED = false>
cudaError_t launch_one(const FwdLaunch& l, cudaStream_t stream) {
  const bool one_tile = one_tile_per_cta<D, CAUSAL, DROPOUT>(l);
  if constexpr (!DROPOUT) {
    if (rows_layout<D, DROPOUT>(l))
      return one_tile ? launch_groups<D, BF16, CAUSAL, DROPOUT, BS, 1, true, PADDED>(l, stream)
                      : launch_groups<D, BF16, CAUSAL, DROPOUT, BS, 2, true, PADDED>(l, stream);
  }
  if constexpr (D == 64 || DROPOUT) {
    return one_tile ? launch_groups<D, BF16, CAUSAL, DROPOUT, BS, 1, false, PADDED>(l, stream)
                    : launch_groups<D, BF16, CAUSAL, DROPOUT, BS, 2, false, PADDED>(l, stream);
  }
  return cudaErrorInvalidValue;
}

template <int D, bool BF16, bool CAUSAL>
cudaError_t launch_dd(const FwdLaunch& l, cudaStream_t stream) {
  return l.is_dropout ? launch_one<D, BF16, CAUSAL, true, false>(l, stream)
                      : launch_one<D, BF16, CAUSAL, false, false>(l, stream);
}

template <int D>
cudaError_t launch_d(const FwdLaunch& l, cudaStream_t stream) {
  if (l.is_bf16) {
    return l.is_causal ? launch_dd<D, true, true>(l, stream) : launch_dd<D, true, false>(l, stream);
  }
  return l.is_causal ? launch_dd<D, false, true>(l, stream) : launch_dd<D, false, false>(l, stream);
}

}  // namespace

int out_box_columns(const FwdLaunch& l) {
  if (l.dpad == 64) {
    if (l.is_causal) return l.is_dropout ? box_columns<64, true, true>(l) : box_columns<64, true, false>(l);
    return l.is_dropout ? box_columns<64, false, true>(l) : box_columns<64, false, false>(l);
  }
  if (l.is_causal) return l.is_dropout ? box_columns<128, true, true>(l) : box_columns<128, true, false>(l);
  return l.is_dropout ? box_columns<128, false, true>(l) : box_columns<128, false, false>(l);
}

cudaError_t launch_fwd(const FwdLaunch& l, cudaStream_t stream) {
  if (l.args.bs_iter != nullptr) {
    // block-sparse exists for fp16 and head_dim <= 64 (checked by the C ABI)
    if (l.is_causal)
      return l.is_dropout ? launch_one<64, false, true, true, true>(l, stream)
                          : launch_one<64, false, true, false, true>(l, stream);
    return l.is_dropout ? launch_one<64, false, false, true, true>(l, stream)
                        : launch_one<64, false, false, false, true>(l, stream);
  }
  return l.dpad == 64 ? launch_d<64>(l, stream) : launch_d<128>(l, stream);
}

cudaError_t launch_fwd_padded(const FwdLaunch& l, cudaStream_t stream) {
  if (l.is_bf16 || l.is_dropout || l.args.bs_iter != nullptr) return cudaErrorInvalidValue;
  if (l.dpad == 64)
    return l.is_causal ? launch_one<64, false, true, false, false, true>(l, stream)
                       : launch_one<64, false, false, false, false, true>(l, stream);
  return l.is_causal ? launch_one<128, false, true, false, false, true>(l, stream)
                     : launch_one<128, false, false, false, false, true>(l, stream);
}

}  // namespace fa
