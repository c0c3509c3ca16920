// FlashAttention backward for sm_100a.
//
// Three launches:
//   1. bwd_preprocess: softmax_d[b,h,i] = p_keep * sum_d dO*O and zero-fill of the fp32 dQ
//      accumulator (HBM bound).
//   2. bwd_main: a block per 128-row key/value tile of one (batch, head) pair, worked on by a CTA of its own or, where
//      there are more blocks than SMs, by one that takes over one block after the other; it keeps K and V in
//      shared memory and walks the 128-row query tiles.  Per tile pair it recomputes
//      S = Q K^T and dP = dO V^T on the tensor cores (accumulators in tensor memory), forms
//      P = exp2(scale*log2e*S - LSE*log2e), regenerates the dropout mask, forms
//      dS = P*(dP - D) (kept) or -P*D (dropped), writes the 16-bit P~ and dS to shared memory
//      and issues dV += P~^T dO, dK += dS^T Q, dQ = dS K.  dQ tiles are added into the fp32
//      accumulator with TMA reduce-adds; dK and dV stay in tensor memory until the end.
//   3. bwd_postprocess: dq = accumulator * scale / p_keep in the 16-bit output type.
//
// The formulas are those of the reference backward
// (csrc/flash_attn/src/fmha_dgrad_kernel_1xN_loop.h:304-661): P recomputed from the saved LSE
// (:333), dropped entries contribute -P*D (:402-418), dQ and dK scaled by scale/p_keep (:583,
// :628), dV by 1/p_keep (:613-619), P~ and dS rounded to the 16-bit type before their products.
//
// Warp roles in bwd_main:
//   compute     eight warps (sixteen at d = 64 with dropout): S, dP -> P~, dS.  Eight: warps 0-3 take key columns 0-63
//               of the tile, warps 4-7 the others, one thread per query row.  Sixteen: a 16-row block and one half of
//               the columns each, in the 16x256b quad layout in which one Philox call is private to a thread, with
//               stmatrix stores; four warps per scheduler cover each other's generator chains and waits.  Main kernel,
//               us, eight -> sixteen (a CTA per block): 8 x 12 x 4096 ragged 1037 -> 944, causal 8 x 12 x 2048 255 -> 245,
//               8 x 16 x 1000 (d = 32) 110 -> 104, 32 x 12 x 200 50.8 -> 49.9.
//   then four   dQ group: tensor memory -> global reductions
//   last four   TMA producer, MMA issuer (S, dP, dQ; everything at d = 128), second and third issuer (dV | dK) at d = 64
// The compute warps write dV and dK at the end.
//
// Schedules.  d = 64: Q and dO travel together through a three-stage ring (two stages for block-sparse calls, and for few queries, which
// hold two stages of K and V instead: short_queries in fa_rules.h); S and dP of tile t + 1 are issued as soon as the compute groups have read tile t into registers.  d = 128: shared
// memory holds one stage of Q and one of dO, each with its own barriers.  The compute groups work
// in two phases, P~ from S and then dS from dP; dV(t) is issued after phase one and releases dO
// for its refill, dK(t) and dQ(t) follow phase two and dK releases Q; S(t + 1) is issued when Q
// has landed and dP(t + 1) when dO has landed and the dQ group has read dQ(t) out of the
// tensor-memory columns it shares with dP.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <type_traits>
#include "fa_rules.h"
#include "fa_math.cuh"
#include "sm100_prims.cuh"

namespace fa {

namespace {

constexpr int kBM = 128;  // query rows per tile
constexpr int kBN = 128;  // key rows per tile
constexpr int kMaxSparseTiles = 1024;  // query tiles of 128 per sequence in block-sparse mode

// BS: block-sparse variant (its tile list takes shared memory that the third Q / dO stage would need)
// SHORT: see short_queries
template <int D, bool BS = false, bool DROPOUT = false, bool SHORT = false>
struct BwdCfg {
  // d = 128 runs a different schedule: shared memory holds a single stage of Q and of dO, each
  // with its own barriers, and the compute groups work in two phases (P~ from S, then dS from dP)
  // so that dV can be issued - and dO released for its refill - before dP is even needed.
  static constexpr bool kTwoPhase = (D == 128);
  // Q / dO ring.  d = 64: a stage is released when the dK product of its tile has finished and
  // the refill takes about 1500 clk to land, so with two stages the S / dP products of the next
  // tile start late and the compute groups wait; the third stage lets the load run a whole tile
  // ahead.
  static constexpr int kQStages = (D == 64) ? (BS || SHORT ? 2 : 3) : 1;
  static constexpr int kKvStages = SHORT ? 2 : 1;
  // Compute warps.  d = 64 with dropout: sixteen of one 16-row block and one half of the keys each (quad layout), four
  // per scheduler, which cover each other's waits and generator chains; else eight, a thread per row and half.
  static constexpr bool kQuad = DROPOUT && !kTwoPhase;
  static constexpr int kComputeWarps = kQuad ? 16 : 8;
  static constexpr int kThreads = 32 * kComputeWarps + 256;  // + the dQ group, + producer and issuers
  // register split (per thread) of the 128 (80 with sixteen compute warps) a thread is launched with
  static constexpr int kComputeRegs = kQuad ? 96 : kTwoPhase ? 168 : 184;
  static constexpr int kDqRegs = kQuad ? 64 : kTwoPhase ? 104 : 88;
  static constexpr int kOtherRegs = kQuad ? 32 : kTwoPhase ? 72 : 56;
  // arrivals of the compute warps at a barrier: every thread, or one lane per warp
  static constexpr uint32_t kComputeArrivals = kQuad ? 16 : 256;
  static constexpr bool kAliasDq = kTwoPhase;     // dQ shares tensor-memory columns with dP
  static constexpr bool kDualIssue = !kTwoPhase;  // second MMA-issuing warp for dV, dK
  static constexpr int kTileBytes = 128 * D * 2;
  static constexpr int kPdsBytes = 128 * 128 * 2;
  static constexpr int kDqStageBytes = 2 * 16384;  // two [128 rows x 32 fp32] boxes
  // (K, V) x stages, (Q, dO) x stages, P~, dS, dQ staging
  static constexpr int kSmemBytes = 2 * (kKvStages + kQStages) * kTileBytes + 2 * kPdsBytes + kDqStageBytes + 1024;
  static constexpr uint32_t kTmemS = 0, kTmemDP = 128, kTmemDV = 256, kTmemDK = 256 + D;
  static constexpr uint32_t kTmemDQ = kAliasDq ? 128 : 256 + 2 * D;
  // A second copy of the 16-bit dS goes to tensor memory and feeds
  // dQ = dS K as the A operand (its M dimension is the query row, like the lanes of S), so that
  // product does not read dS from shared memory; dK = dS^T Q still takes the shared-memory copy.
  // Used without dropout, where shared-memory bandwidth is the bound (d = 64, 8 x 12 x 4096: 1.49 -> 1.39 ms);
  // with dropout the compute groups are the bound and the extra stores cost 2 %.  d = 64 leaves 64 columns free for it; at d = 128 it takes
  // the place of the scores, 32 columns in each half of them: a thread overwrites what it has read itself, and the next S is issued behind dQ.
  // There, us: 4 x 12 x 4096 1155 -> 1147 (causal 607 -> 603), 16 x 12 x 1000 causal 241.7 -> 240.4, back to back under the power
  // limit 16 x 12 x 8192 causal 9860 -> 9817.
  static constexpr uint32_t kTmemDS = kTwoPhase ? kTmemS : 256 + 3 * D;
};

// What a block works on: key tile n0 / 128 of one (batch, head) pair.  nm: query tiles to walk, -1 behind the last block.  The size of the
// record decides how the compiler reads it from shared memory: in 32 bytes two wide loads, best with a causal mask (d = 64, 2 x 4 x
// 16384: 703 us, in 36 bytes 712), in 36 bytes each word where it is used, best without (4 x 12 x 4096 561 and 554 us, ragged batches up to
// 512 tokens with dropout 306 and 303).
template <bool CAUSAL>
struct BlockRecord {
  int q_start, sq, k_start, sk, n0, h, b, nm;
};
template <>
struct BlockRecord<false> {
  int q_start, sq, k_start, sk, n0, h, b, nm, unused;
};
static_assert(sizeof(BlockRecord<true>) == 32 && sizeof(BlockRecord<false>) == 36, "sizes that were measured");

template <bool CAUSAL>
struct BwdShared {
  uint64_t k_full[2], v_full[2], k_empty[2], v_empty[2];  // the key tile's operands, once per key tile
  uint64_t acc_free;                          // dV and dK read out, once per key tile
  uint64_t next_full;                         // the answer to a request for another block is in `next`
  uint64_t blk_full[2], blk_done[2];          // the block after is in `blk`; every role has finished the one there
  uint64_t drained[3];                        // of the issuing warps, at their end
  alignas(16) uint4 next;
  alignas(16) BlockRecord<CAUSAL> blk[2];               // block k in entry k % 2
  uint64_t q_full[3], q_empty[3];
  uint64_t do_full, do_empty;  // dO ring of the two-phase schedule (one stage)
  // d = 64: S and dP together / P~ and dS together.  Two-phase schedule: sdp_full = dP landed,
  // sdp_consumed = S read into registers, pds_ready = dS stored, pds_free = dV has read P~.
  uint64_t sdp_full, sdp_consumed, pds_ready, pds_free, dq_full, dq_consumed;
  uint64_t s_full;    // two-phase: S landed
  uint64_t p_ready;   // two-phase: P~ stored
  uint64_t ds_free;   // two-phase: dK and dQ have finished reading the dS buffer
  uint64_t stat_ready;  // one launch: softmax_d is written
  uint64_t dq_group;  // rendezvous of the 128 threads of the dQ group (bounded, unlike bar.sync)
  uint32_t tmem_base;
  int abort_flag;
};

template <bool BF16>
__device__ __forceinline__ uint32_t pack16(float lo, float hi) {
  if constexpr (BF16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}

// sum of the products of eight 16-bit values, in order
template <bool BF16>
__device__ __forceinline__ float dot8(const uint4& ov, const uint4& gv) {
  const uint32_t ow[4] = {ov.x, ov.y, ov.z, ov.w}, gw[4] = {gv.x, gv.y, gv.z, gv.w};
  float acc = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float2 of, gf;
    if constexpr (BF16) {
      of = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ow[k]));
      gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw[k]));
    } else {
      of = __half22float2(*reinterpret_cast<const __half2*>(&ow[k]));
      gf = __half22float2(*reinterpret_cast<const __half2*>(&gw[k]));
    }
    acc += of.x * gf.x + of.y * gf.y;
  }
  return acc;
}

template <int N>
__device__ __forceinline__ void reg_alloc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void reg_dealloc() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// The three kernels overlap at their ends (programmatic dependent launch): the main kernel's CTAs set up and load their
// first tiles while the last blocks of the preprocess run, and the postprocess is on the SMs when the last main CTA
// leaves.  What a kernel takes from the one before it (softmax_d, the cleared accumulator, tickets | the accumulator) comes behind
// grid_dep_wait, which waits for all of that kernel's blocks and their writes.  Every CTA of the main kernel waits, also one without
// work, so that whatever waits for the main kernel is behind the preprocess too.  Whole backward with its autograd call, us,
// before -> now: 8 x 12 x 512 with dropout 51 -> 49, 16 x 12 x 1024 187 -> 183, 64 x 12 x 512 244 -> 241; the preprocess behind
// whatever is ahead of it: training passes of 16 x 8 heads, 200 queries, 1500 keys 80.6 -> 78.4, 8 x 12 x 512 67.6 -> 66.4.
// A launch of this kind takes the host longer, so grids that leave SMs idle, whose calls wait for the host, keep ordinary ones
// (8 x 12 x 128: 21.5 -> 25.8).
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

bool overlap_launches(const BwdLaunch& l) {
  return l.stage_mask == 0 && !l.args.one_launch &&
         static_cast<int64_t>((l.args.max_seqlen_k + kBN - 1) / kBN) * l.args.k.heads * l.args.k.batch > kSms;
}

template <typename... P, typename... A>
cudaError_t launch(bool overlap, void (*kernel)(P...), dim3 grid, int threads, int smem, cudaStream_t stream, const A&... args) {
  if (!overlap) {
    kernel<<<grid, threads, smem, stream>>>(args...);
    return cudaGetLastError();
  }
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// ------------------------------------------------------------------------------------------------
// ONE_LAUNCH: see one_launch()
template <int D, bool BF16, bool CAUSAL, bool DROPOUT, bool BLOCKSPARSE, bool ONE_LAUNCH, bool SHORT>
__global__ void __launch_bounds__(BwdCfg<D, BLOCKSPARSE, DROPOUT, SHORT>::kThreads, 1)
fa_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
              const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
              const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_dk,
              const __grid_constant__ CUtensorMap tm_dv, const BwdArgs a) {
  using Cfg = BwdCfg<D, BLOCKSPARSE, DROPOUT, SHORT>;
  constexpr int kDqWarp = Cfg::kComputeWarps, kProducer = kDqWarp + 4;  // first warp of the dQ group, of the last four
  constexpr bool kVote = Cfg::kQuad && !ONE_LAUNCH;  // (see mbar_wait_warp)
  constexpr int kBoxColumns = grad_box_columns(D, CAUSAL, DROPOUT);
  constexpr bool kTmaRows = kBoxColumns != 0;
  constexpr bool kDsInTmem = !DROPOUT;
  extern __shared__ uint8_t smem_raw[];
  using BlockInfo = BlockRecord<CAUSAL>;
  __shared__ BwdShared<CAUSAL> sh;

  const int tid = threadIdx.x;
  // Known to be the same in all lanes, for the issuing warps (see mma_ss).  The compute and dQ groups take
  // theirs anew and the epilogue works from tid: with one value kept live across all roles short
  // calls at d = 64 lost 1-3 % to lane-0 issue, and spill loads there went from 24 to 76 bytes a thread (32
  // with the values taken anew).  us of the whole backward, lane 0 issuing -> one value -> now: 16 x 8 heads,
  // 200 queries, 1500 keys 79.1 -> 81.2 -> 76.4; 64 x 12 x 512 289 -> 293 -> 271; 2 x 4 x 32768 causal
  // 3632 -> 3309 -> 3226.
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const KernelArgs& ka = a.k;
  // One CTA per SM takes over one block of the grid after the other (cluster launch control, in the order of the grid):
  // the next key tile's operands load and its first products run while dV, dK and the last dQ tiles of the one before
  // leave, instead of after its CTA's end and the start of another, which cost about two query tiles per
  // key tile.  Every role walks the same blocks; c counts the key tiles with work, g the query tiles walked so far,
  // which give the phases of the barriers.  Main kernel, us, a CTA per block -> now: 16 x 8 heads, 200 queries, 1500
  // keys 72.5 -> 52.5; 64 x 12 x 512 227 -> 170; 16 x 12 x 1000 causal (d = 128) 249 -> 205; 8 x 12 x 512 with dropout
  // 41.6 -> 36.9; 2 x 4 x 16384 causal 711 -> 689; 4 x 12 x 8192 causal (d = 128) 2199 -> 2131.  Block-sparse, whole backward, 4 x
  // 16 x 4096 with 25 % of the blocks 398 -> 334, with dropout 442 -> 385, 16 x 12 x 2048 ragged 260 -> 199.
  auto decode = [&](uint32_t block) -> BlockInfo {
    BlockInfo x;
    int nt;
    if (CAUSAL && gridDim.y == 1 && gridDim.z == 1) {
      causal_block(ka, block, nt, x.h, x.b);
    } else if (a.take_over) {
      const uint32_t pair = block / ka.grid_tiles;
      nt = block - pair * ka.grid_tiles;
      x.b = pair / ka.heads;
      x.h = pair - x.b * ka.heads;
    } else {
      nt = blockIdx.x; x.h = blockIdx.y; x.b = blockIdx.z;
    }
    x.q_start = ka.cu_seqlens_q[x.b];
    x.sq = ka.cu_seqlens_q[x.b + 1] - x.q_start;
    x.k_start = ka.cu_seqlens_k[x.b];
    x.sk = ka.cu_seqlens_k[x.b + 1] - x.k_start;
    x.n0 = nt * kBN;
    if constexpr (!CAUSAL) x.unused = 0;
    const int m_tiles = (x.sq + kBM - 1) / kBM;
    // (a call of one launch also writes dq = 0 for a sequence without keys)
    x.nm = x.n0 < x.sk || ONE_LAUNCH ? m_tiles - (CAUSAL ? min(m_tiles, x.n0 / kBM) : 0) : 0;
    return x;
  };
  grid_dep_launch();
  const int32_t failed = ka.status ? *reinterpret_cast<volatile int32_t*>(ka.status) : 0;  // on its way beside the lengths
  BlockInfo first = decode(blockIdx.x);
  // (not in the deterministic mode, whose blocks wait for blocks of smaller index: those start first only as the
  // hardware launches them; and not where every block has an SM at once)
  const bool take_over = a.take_over;
  // a block behind its sequence's last key.  A CTA of its own leaves here, before it takes tensor memory and sets up its
  // barriers: 1 x 4096 and 63 x 128, 12 heads, deterministic, us, through the whole kernel -> here: 869 -> 642 (d = 64),
  // 1311 -> 1044 (d = 128)
  // Whoever leaves early waits for the preprocess too: the postprocess waits for this kernel alone, and a grid whose CTAs all left
  // without a wait could end before the accumulator is cleared.
  if (!take_over && first.n0 >= first.sk && !ONE_LAUNCH) {
    grid_dep_wait();
    return;
  }
  // fail fast: once a CTA of this launch has abandoned a wait, the blocks that have not started do not, whether a CTA of
  // their own or one that takes them over looks
  auto launch_failed = [&]() -> bool {
    return ka.status && *reinterpret_cast<volatile int32_t*>(ka.status) == ka.launch_id;
  };
  if (failed == ka.launch_id) {
    grid_dep_wait();
    return;
  }

  // Block-sparse: the query tiles that have at least one 16-row block in this key block's list, in ascending order; those of block k
  // in list k % 2.  The whole CTA makes the first list, the producer's warp those of blocks taken over.
  constexpr int kListTiles = BLOCKSPARSE ? kMaxSparseTiles : 1;
  __shared__ uint16_t qtile_list[BLOCKSPARSE ? 2 : 1][kListTiles];
  // deterministic mode: how many key tiles before this one add into the same query tile
  __shared__ uint16_t qtile_order[kListTiles];
  __shared__ uint32_t qtile_bits[(kListTiles + 31) / 32];
  // a bit for each of the query tiles [32 c, 32 c + 32) of key block kb (one warp)
  auto list_bits = [&](const BlockInfo& x, int kb, int c, int mt) -> uint32_t {
    const int m = c * 32 + lane, rb_end = min(ka.bs_rows16, (x.sq + 15) >> 4);
    const int32_t* brow = ka.bs_iter + (static_cast<int64_t>(x.b) * ka.bs_kblocks + kb) * ka.bs_rows16;
    bool any = false;
    if (m < mt && !(CAUSAL && m < x.n0 / kBM))  // (query tiles entirely before this key tile see none of it)
#pragma unroll
      for (int i = 0; i < kBM / 16; ++i)
        if (m * (kBM / 16) + i < rb_end) any = any || (brow[m * (kBM / 16) + i] >= 0);
    return __ballot_sync(0xffffffffu, any);
  };
  auto list_tiles = [&](const BlockInfo& x) -> int { return min((x.sq + kBM - 1) / kBM, kMaxSparseTiles); };
  auto put_in_list = [&](uint16_t* list, int c, uint32_t bits, int before) {
    if (bits >> lane & 1) list[before + __popc(bits & ((1u << lane) - 1))] = static_cast<uint16_t>(c * 32 + lane);
  };
  if constexpr (BLOCKSPARSE) {
    const int mt = list_tiles(first);
    for (int c = warp; c * 32 < mt; c += Cfg::kThreads / 32) {
      const uint32_t bits = list_bits(first, first.n0 >> 8, c, mt);
      if (lane == 0) qtile_bits[c] = bits;
    }
    __syncthreads();
    int total = 0;
    for (int c = 0; c * 32 < mt; ++c) {
      const uint32_t bits = qtile_bits[c];
      if (c % (Cfg::kThreads / 32) == warp) {
        put_in_list(qtile_list[0], c, bits, total);
        if (a.dq_tickets != nullptr) {
          // the two 128-row key tiles of a 256-row key block visit the same query tiles
          int before = 0;
          for (int kb = 0; kb < first.n0 >> 8; ++kb) before += (list_bits(first, kb, c, mt) >> lane & 1) * 2;
          if (bits >> lane & 1)
            qtile_order[total + __popc(bits & ((1u << lane) - 1))] = static_cast<uint16_t>(before + (first.n0 / kBN & 1));
        }
      }
      total += __popc(bits);
    }
    first.nm = first.n0 < first.sk ? total : 0;  // (the list is read behind the barrier below)
  }
  // Deterministic mode: the key tiles of one (batch, head) add into a query tile in ascending
  // key-tile order.  Dense causal grids then walk the query tiles from the last one down, so that
  // every key tile starts on a query tile its predecessors start on too (walking up, key tile n
  // would idle until tile n - 1 arrives at its first query tile).
  const bool deterministic = a.dq_tickets != nullptr;
  const bool walk_down = CAUSAL && !BLOCKSPARSE && deterministic;
  auto q_tile = [&](const BlockInfo& x, int t, uint32_t k) -> int {  // of block k
    if constexpr (BLOCKSPARSE) return qtile_list[k & 1][t];
    const int m_tiles = (x.sq + kBM - 1) / kBM;
    return walk_down ? m_tiles - 1 - t : m_tiles - x.nm + t;  // causal: from the tile of the first key on
  };

  uint16_t* dk_base = reinterpret_cast<uint16_t*>(a.dk);
  uint16_t* dv_base = reinterpret_cast<uint16_t*>(a.dv);

  // no query row sees these keys: their gradients are zero (`threads` threads from thread 0 on)
  auto zero_tile = [&](const BlockInfo& x, int threads) {
    for (int idx = tid; idx < kBN * (ka.head_dim / 8); idx += threads) {
      const int r = idx / (ka.head_dim / 8), c = (idx % (ka.head_dim / 8)) * 8;
      if (x.n0 + r < x.sk) {
        const int64_t row = x.k_start + x.n0 + r;
        *reinterpret_cast<uint4*>(dk_base + row * a.dk_row_stride + x.h * a.dk_head_stride + c) =
            make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(dv_base + row * a.dv_row_stride + x.h * a.dv_head_stride + c) =
            make_uint4(0, 0, 0, 0);
      }
    }
  };

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const uint32_t smem_k = smem_u32(smem);
  const uint32_t smem_v = smem_k + Cfg::kTileBytes;  // of the first stage
  auto kv_at = [&](int c) -> uint32_t { return c % Cfg::kKvStages * (2 * Cfg::kTileBytes); };  // of key tile c
  const uint32_t smem_q = smem_k + 2 * Cfg::kKvStages * Cfg::kTileBytes;  // stages of Q
  const uint32_t smem_do = smem_q + Cfg::kQStages * Cfg::kTileBytes;      // stages of dO
  const uint32_t smem_p = smem_do + Cfg::kQStages * Cfg::kTileBytes;
  const uint32_t smem_ds = smem_p + Cfg::kPdsBytes;
  uint8_t* p_ptr = smem + 2 * (Cfg::kKvStages + Cfg::kQStages) * Cfg::kTileBytes;
  uint8_t* ds_ptr = p_ptr + Cfg::kPdsBytes;
  uint8_t* dq_stage = ds_ptr + Cfg::kPdsBytes;

  if (tid == 0) {
    sh.abort_flag = 0;
    for (int i = 0; i < Cfg::kKvStages; ++i) {
      mbar_init(smem_u32(&sh.k_full[i]), 1);
      mbar_init(smem_u32(&sh.v_full[i]), 1);
      mbar_init(smem_u32(&sh.k_empty[i]), 1);
      mbar_init(smem_u32(&sh.v_empty[i]), 1);
    }
    mbar_init(smem_u32(&sh.stat_ready), 4);
    mbar_init(smem_u32(&sh.acc_free), Cfg::kComputeWarps);
    mbar_init(smem_u32(&sh.next_full), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&sh.blk_full[i]), 1);
      mbar_init(smem_u32(&sh.blk_done[i]), Cfg::kComputeWarps + 4 + (Cfg::kDualIssue ? 3 : 1));  // all but the producer
    }
    sh.blk[0] = first;
    for (int i = 0; i < 3; ++i) {
      mbar_init(smem_u32(&sh.drained[i]), 1);
      mbar_init(smem_u32(&sh.q_full[i]), 1);
      mbar_init(smem_u32(&sh.q_empty[i]), Cfg::kDualIssue ? 2 : 1);  // d = 64: dV (reads dO) and dK (reads Q)
    }
    mbar_init(smem_u32(&sh.do_full), 1);
    mbar_init(smem_u32(&sh.do_empty), 1);
    mbar_init(smem_u32(&sh.sdp_full), 1);
    mbar_init(smem_u32(&sh.sdp_consumed), Cfg::kComputeArrivals);
    mbar_init(smem_u32(&sh.pds_ready), Cfg::kComputeArrivals);
    mbar_init(smem_u32(&sh.pds_free), Cfg::kDualIssue ? 3 : 1);  // d = 64: dQ, dV and dK each commit
    mbar_init(smem_u32(&sh.dq_full), 1);
    mbar_init(smem_u32(&sh.dq_consumed), kBM);
    mbar_init(smem_u32(&sh.dq_group), kBM);
    mbar_init(smem_u32(&sh.s_full), 1);
    mbar_init(smem_u32(&sh.p_ready), Cfg::kComputeArrivals);
    mbar_init(smem_u32(&sh.ds_free), 1);
    fence_mbar_init();
  }
  if (warp == kProducer) tmem_alloc(smem_u32(&sh.tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem_base;
  volatile int* abort_flag = &sh.abort_flag;

  const float rp_keep = ka.rp_keep;

  // operand descriptors of the five products
  constexpr uint32_t idesc_s = make_idesc(BF16, false, false, 128, 128);   // Q K^T, dO V^T
  constexpr uint32_t idesc_tt = make_idesc(BF16, true, true, 128, D);      // P~^T dO, dS^T Q
  constexpr uint32_t idesc_dq = make_idesc(BF16, false, true, 128, D);     // dS K
  // Called by one elected lane of an issuing warp whose lanes all run the surrounding loop (see mma_ss).
  auto issue_kk = [&](uint32_t dst, uint32_t a_base, uint32_t b_base) {  // both K-major, K = D
    const uint64_t da = desc_here(make_smem_desc(a_base, 16, 1024)), db = desc_here(make_smem_desc(b_base, 16, 1024));
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      const uint32_t off = (ks >> 2) * 16384 + (ks & 3) * 32;
      mma_ss(dst, desc_at(da, off), desc_at(db, off), idesc_s, ks > 0);
    }
  };
  auto issue_tt = [&](uint32_t dst, uint32_t a_base, uint32_t b_base, bool acc) {
    // A = [q][kv] read as M = kv (MN-major); B = [q][d] read as N = d (MN-major); K = q rows
    const uint64_t da = desc_here(make_smem_desc(a_base, 16384, 1024)), db = desc_here(make_smem_desc(b_base, 16384, 1024));
#pragma unroll
    for (int ks = 0; ks < kBM / 16; ++ks)
      mma_ss(dst, desc_at(da, ks * 2048), desc_at(db, ks * 2048), idesc_tt, acc || ks > 0);
  };
  auto issue_dq = [&](uint32_t dst, uint32_t a_base, uint32_t b_base) {
    // A = dS [q][kv] K-major; B = K [kv][d] read as N = d (MN-major); K = kv
    const uint64_t da = desc_here(make_smem_desc(a_base, 16, 1024)), db = desc_here(make_smem_desc(b_base, 16384, 1024));
#pragma unroll
    for (int ks = 0; ks < kBN / 16; ++ks) {
      const uint32_t off = (ks >> 2) * 16384 + (ks & 3) * 32;
      mma_ss(dst, desc_at(da, off), desc_at(db, ks * 2048), idesc_dq, ks > 0);
    }
  };
  const uint32_t tS_ = tmem + Cfg::kTmemS, tDP_ = tmem + Cfg::kTmemDP;
  const uint32_t tDV_ = tmem + Cfg::kTmemDV, tDK_ = tmem + Cfg::kTmemDK, tDQ_ = tmem + Cfg::kTmemDQ;
  const uint32_t tDS_ = tmem + Cfg::kTmemDS;
  auto issue_dq_t = [&](uint32_t dst, uint32_t a_tmem, uint32_t b_base) {
    // A = dS from tensor memory (16 keys = 8 columns per step); B = K [kv][d] read as N = d; K = kv
    const uint64_t db = desc_here(make_smem_desc(b_base, 16384, 1024));
#pragma unroll
    for (int ks = 0; ks < kBN / 16; ++ks)
      mma_ts(dst, a_tmem + (Cfg::kTwoPhase ? (ks >> 2) * 64 + (ks & 3) * 8 : ks * 8), desc_at(db, ks * 2048), idesc_dq, ks > 0);
  };

  // A warp has finished block k: waits for the next one, if any (or until a wait is abandoned).
  auto next_block = [&](uint32_t k) -> bool {
    if (!take_over) return false;
    __syncwarp();
    if (elect_one()) mbar_arrive(smem_u32(&sh.blk_done[k & 1]));
    return mbar_wait_warp<kVote>(smem_u32(&sh.blk_full[(k + 1) & 1]), (k >> 1) & 1, abort_flag) && sh.blk[(k + 1) & 1].nm >= 0;
  };

  if (warp >= kProducer) {
    reg_dealloc<Cfg::kOtherRegs>();
    if (warp == kProducer && (BLOCKSPARSE || lane == 0)) {
      // -------------------------------------------------------------- TMA producer
      // (one lane; block-sparse: the warp stays together, to make the lists of blocks taken over, and one lane issues)
      const bool lead = !BLOCKSPARSE || lane == 0;
      auto wait = [&](uint64_t& bar, uint32_t parity) -> bool {
        const bool done = mbar_wait(smem_u32(&bar), parity, abort_flag);
        return BLOCKSPARSE ? __all_sync(0xffffffffu, done) : done;
      };
      auto load = [&](uint32_t dst, const CUtensorMap* map, uint64_t& bar, int row, int h) {
        for (int p = 0; p < D / 64; ++p) tma_load_3d(dst + p * 16384, map, smem_u32(&bar), p * 64, row, h);
      };
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      tma_prefetch_desc(&tm_do);
      if constexpr (!ONE_LAUNCH) tma_prefetch_desc(&tm_dq);
      bool ok = true;
      int loads_k = 0, loads_v = 0, loads_q = 0, loads_do = 0;  // so far
      uint32_t asked = 0;                                       // requests so far
      BlockInfo x = sh.blk[0];
      for (uint32_t k = 0; ok; ++k) {
        const int nm = x.nm, h = x.h;
        // asked for when the last query tile is under way: a block taken earlier would wait here while other SMs run dry
        auto take_next = [&]() {
          if (!take_over) return;
          if (lead) {
            mbar_expect_tx(smem_u32(&sh.next_full), 16);
            clc_try_cancel(smem_u32(&sh.next), smem_u32(&sh.next_full));
          }
          ++asked;
        };
        if (nm <= 0) take_next();
        for (int t = 0; t < nm && ok; ++t) {
          const int s = loads_q % Cfg::kQStages;
          const int row = x.q_start + q_tile(x, t, k) * kBM;
          auto load_k = [&]() {
            const int stage = loads_k % Cfg::kKvStages;
            if (loads_k >= Cfg::kKvStages) ok = wait(sh.k_empty[stage], ((loads_k / Cfg::kKvStages) & 1) ^ 1);
            if (!ok) return;
            if (lead) {
              mbar_expect_tx(smem_u32(&sh.k_full[stage]), Cfg::kTileBytes);
              load(smem_k + kv_at(loads_k), &tm_k, sh.k_full[stage], x.k_start + x.n0, h);
            }
            ++loads_k;
          };
          const bool first_k = t == 0 && (SHORT || loads_k == 0);
          if (first_k) load_k();
          if (t == 0) {
            // V is free after the last dP of the key tile before, K after its last dQ
            const int stage = loads_v % Cfg::kKvStages;
            if (ok && loads_v >= Cfg::kKvStages) ok = wait(sh.v_empty[stage], ((loads_v / Cfg::kKvStages) & 1) ^ 1);
            if (!ok) break;
            if (lead) {
              mbar_expect_tx(smem_u32(&sh.v_full[stage]), Cfg::kTileBytes);
              load(smem_v + kv_at(loads_v), &tm_v, sh.v_full[stage], x.k_start + x.n0, h);
            }
            ++loads_v;
          }
          if constexpr (Cfg::kTwoPhase) {
            // dO(g) follows dV(g - 1), Q(g) follows dK(g - 1): the order in which they finish
            if (loads_do > 0) ok = wait(sh.do_empty, (loads_do & 1) ^ 1);
            if (!ok) break;
            mbar_expect_tx(smem_u32(&sh.do_full), Cfg::kTileBytes);
            load(smem_do, &tm_do, sh.do_full, row, h);
            ++loads_do;
            if (loads_q > 0) ok = wait(sh.q_empty[0], (loads_q & 1) ^ 1);
            if (!ok) break;
            mbar_expect_tx(smem_u32(&sh.q_full[0]), Cfg::kTileBytes);
            load(smem_q, &tm_q, sh.q_full[0], row, h);
          } else {
            if (loads_q >= Cfg::kQStages)
              ok = wait(sh.q_empty[s], ((loads_q / Cfg::kQStages) & 1) ^ 1);
            if (!ok) break;
            if (lead) {
              mbar_expect_tx(smem_u32(&sh.q_full[s]), 2 * Cfg::kTileBytes);
              load(smem_q + s * Cfg::kTileBytes, &tm_q, sh.q_full[s], row, h);
              load(smem_do + s * Cfg::kTileBytes, &tm_do, sh.q_full[s], row, h);
            }
          }
          ++loads_q;
          if (t == 0 && !first_k) load_k();
          if (ok && t + 1 == nm) take_next();
        }
        if (!ok || !take_over) break;
        // The next block with keys.  Those behind their sequence's last key have nothing to do and stay with the producer:
        // passed on, each cost a round through all roles.  us of an SM for such a block, 64 x 12 x 128 announced with 8192
        // keys: a CTA each 0.72, passed on 0.82-0.93, here 0.52-0.65; 1 x 8192 and 31 x 256, 12 heads 771 -> 712 (d = 64).
        bool more = false;
        while (true) {
          ok = wait(sh.next_full, (asked - 1) & 1);
          if (!ok) break;
          uint32_t block;
          more = clc_answer(smem_u32(&sh.next), block);
          fence_async_smem();
          if (!more) break;
          more = !launch_failed();
          if (BLOCKSPARSE) more = __all_sync(0xffffffffu, more);
          x = decode(block);
          if (!more || x.n0 < x.sk || asked % kPassOnEvery == 0) break;  // (the last: see kPassOnEvery)
          take_next();
        }
        if (!ok) break;
        if (!more) x.nm = -1;
        // its place is free once every role has finished block k - 1
        if (k >= 1) ok = wait(sh.blk_done[(k + 1) & 1], ((k - 1) >> 1) & 1);
        if (!ok) break;
        if constexpr (BLOCKSPARSE) {
          if (more && x.n0 < x.sk) {
            const int mt = list_tiles(x);
            x.nm = 0;
            for (int c = 0; c * 32 < mt; ++c) {
              const uint32_t bits = list_bits(x, x.n0 >> 8, c, mt);
              put_in_list(qtile_list[(k + 1) & 1], c, bits, x.nm);
              x.nm += __popc(bits);
            }
          }
          __syncwarp();
        }
        if (lead) {
          sh.blk[(k + 1) & 1] = x;
          mbar_arrive(smem_u32(&sh.blk_full[(k + 1) & 1]));
        }
        if (!more) break;
      }
      mbar_drain_ring(sh.k_full, Cfg::kKvStages, loads_k);
      mbar_drain_ring(sh.v_full, Cfg::kKvStages, loads_v);
      mbar_drain_ring(sh.q_full, Cfg::kQStages, loads_q);
      mbar_drain_ring(&sh.do_full, 1, loads_do);
      mbar_drain_ring(&sh.next_full, 1, asked);
    } else if (warp == kProducer + 1) {
      // -------------------------------------------------------------- MMA issuer 1
      bool ok = true;
      int c = 0, g0 = 0;
      uint32_t k = 0;
      do {
      const int nm = __shfl_sync(0xffffffffu, sh.blk[k & 1].nm, 0);
      if (nm <= 0) continue;
      const int kv = c % Cfg::kKvStages;
      const uint32_t smem_kc = smem_k + kv_at(c), smem_vc = smem_v + kv_at(c);
      ok = mbar_wait_warp<kVote>(smem_u32(&sh.k_full[kv]), (c / Cfg::kKvStages) & 1, abort_flag);
      if constexpr (Cfg::kTwoPhase) {
        // d = 128: every product, issued by this thread in the order
        //   dV(t) | dK(t), dQ(t) | S(t+1) | dP(t+1)
        // dV(t) follows P~ (end of phase one of the compute groups) and releases dO for its
        // refill while phase two is still running.  dK, dQ follow dS; dK releases Q.  S(t+1) is
        // issued when Q has landed, dP(t+1) when dO has landed and the dQ group has read dQ(t)
        // out of the columns it shares with dP.
        auto scores = [&](int g) {
          ok = mbar_wait_warp(smem_u32(&sh.q_full[0]), g & 1, abort_flag);
          if (ok && g > 0) ok = mbar_wait_warp(smem_u32(&sh.sdp_consumed), (g & 1) ^ 1, abort_flag);
          if (!ok) return;
          tc_fence_after();
          if (elect_one()) {
            issue_kk(tS_, smem_q, smem_kc);
            mma_commit(smem_u32(&sh.s_full));
          }
        };
        auto grad_p = [&](int g, bool last) {
          ok = mbar_wait_warp(smem_u32(&sh.do_full), g & 1, abort_flag);
          if (ok && g > 0) ok = mbar_wait_warp(smem_u32(&sh.dq_consumed), (g & 1) ^ 1, abort_flag);
          if (!ok) return;
          tc_fence_after();
          if (elect_one()) {
            issue_kk(tDP_, smem_do, smem_vc);
            mma_commit(smem_u32(&sh.sdp_full));
            if (last) mma_commit(smem_u32(&sh.v_empty[kv]));
          }
        };
        if (ok) scores(g0);
        if (ok) ok = mbar_wait_warp(smem_u32(&sh.v_full[kv]), (c / Cfg::kKvStages) & 1, abort_flag);
        if (ok) grad_p(g0, nm == 1);
        for (int t = 0; t < nm && ok; ++t) {
          const int g = g0 + t;
          const bool has_next = t + 1 < nm;
          if (t == 0 && c > 0) {
            ok = mbar_wait_warp(smem_u32(&sh.acc_free), (c & 1) ^ 1, abort_flag);
            if (!ok) break;
          }
          ok = mbar_wait_warp(smem_u32(&sh.p_ready), g & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_tt(tDV_, smem_p, smem_do, t > 0);
            mma_commit(smem_u32(&sh.pds_free));
            mma_commit(smem_u32(&sh.do_empty));
          }
          ok = mbar_wait_warp(smem_u32(&sh.pds_ready), g & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_tt(tDK_, smem_ds, smem_q, t > 0);
            mma_commit(smem_u32(&sh.q_empty[0]));
            if constexpr (kDsInTmem) issue_dq_t(tDQ_, tDS_, smem_kc);
            else issue_dq(tDQ_, smem_ds, smem_kc);
            mma_commit(smem_u32(&sh.dq_full));
            mma_commit(smem_u32(&sh.ds_free));
            if (!has_next) mma_commit(smem_u32(&sh.k_empty[kv]));
          }
          if (has_next) {
            scores(g + 1);
            if (ok) grad_p(g + 1, t + 2 == nm);
          }
        }
      } else {
        // d = 64: S, dP and dQ (dV, dK go through issuer 2)
        auto scores = [&](int g, bool last) {
          const int s = g % Cfg::kQStages;
          ok = mbar_wait_warp<kVote>(smem_u32(&sh.q_full[s]), (g / Cfg::kQStages) & 1, abort_flag);
          if (ok && g > 0) ok = mbar_wait_warp<kVote>(smem_u32(&sh.sdp_consumed), (g & 1) ^ 1, abort_flag);
          if (!ok) return;
          tc_fence_after();
          if (elect_one()) {
            issue_kk(tS_, smem_q + s * Cfg::kTileBytes, smem_kc);
            issue_kk(tDP_, smem_do + s * Cfg::kTileBytes, smem_vc);
            mma_commit(smem_u32(&sh.sdp_full));
            if (last) mma_commit(smem_u32(&sh.v_empty[kv]));
          }
        };
        if (ok) ok = mbar_wait_warp<kVote>(smem_u32(&sh.v_full[kv]), (c / Cfg::kKvStages) & 1, abort_flag);
        if (ok) scores(g0, nm == 1);
        for (int t = 0; t < nm && ok; ++t) {
          const int g = g0 + t;
          if (t + 1 < nm) scores(g + 1, t + 2 == nm);
          if (ok) ok = mbar_wait_warp<kVote>(smem_u32(&sh.pds_ready), g & 1, abort_flag);
          if (ok && g > 0) ok = mbar_wait_warp<kVote>(smem_u32(&sh.dq_consumed), (g & 1) ^ 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          // its tile is read out of tensor memory while dV / dK are still running
          if (elect_one()) {
            if constexpr (kDsInTmem) issue_dq_t(tDQ_, tDS_, smem_kc);
            else issue_dq(tDQ_, smem_ds, smem_kc);
            mma_commit(smem_u32(&sh.dq_full));
            mma_commit(smem_u32(&sh.pds_free));
            if (t + 1 == nm) mma_commit(smem_u32(&sh.k_empty[kv]));
          }
        }
      }
      ++c;
      g0 += nm;
      } while (ok && next_block(k++));
      mma_drain(smem_u32(&sh.drained[0]));
    } else if (warp == kProducer + 2 && Cfg::kDualIssue) {
      // -------------------------------------------------------------- MMA issuer 2: dV
      // dV and dK have a warp each, so that neither waits for the other's instructions to be taken.
      bool ok = true;
      int c = 0, g = 0;
      uint32_t k = 0;
      do {
        const int nm = __shfl_sync(0xffffffffu, sh.blk[k & 1].nm, 0);
        if (nm <= 0) continue;
        if (c > 0) ok = mbar_wait_warp<kVote>(smem_u32(&sh.acc_free), (c & 1) ^ 1, abort_flag);
        for (int t = 0; t < nm && ok; ++t, ++g) {
          const int s = g % Cfg::kQStages;
          ok = mbar_wait_warp<kVote>(smem_u32(&sh.pds_ready), g & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_tt(tDV_, smem_p, smem_do + s * Cfg::kTileBytes, t > 0);
            mma_commit(smem_u32(&sh.pds_free));
            mma_commit(smem_u32(&sh.q_empty[s]));
          }
        }
        ++c;
      } while (ok && next_block(k++));
      mma_drain(smem_u32(&sh.drained[1]));
    } else if (warp == kProducer + 3 && Cfg::kDualIssue) {
      // -------------------------------------------------------------- MMA issuer 3: dK
      bool ok = true;
      int c = 0, g = 0;
      uint32_t k = 0;
      do {
        const int nm = __shfl_sync(0xffffffffu, sh.blk[k & 1].nm, 0);
        if (nm <= 0) continue;
        if (c > 0) ok = mbar_wait_warp<kVote>(smem_u32(&sh.acc_free), (c & 1) ^ 1, abort_flag);
        for (int t = 0; t < nm && ok; ++t, ++g) {
          const int s = g % Cfg::kQStages;
          ok = mbar_wait_warp<kVote>(smem_u32(&sh.pds_ready), g & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_tt(tDK_, smem_ds, smem_q + s * Cfg::kTileBytes, t > 0);
            mma_commit(smem_u32(&sh.pds_free));
            mma_commit(smem_u32(&sh.q_empty[s]));
          }
        }
        ++c;
      } while (ok && next_block(k++));
      mma_drain(smem_u32(&sh.drained[2]));
    }
  } else if (warp < kDqWarp) {
    // ------------------------------------------------------------------ compute groups
    // group w (0 / 1) owns key columns [64 w, 64 w + 64) of the tile; one thread per query row
    reg_alloc<Cfg::kComputeRegs>();
    grid_dep_wait();
    const int cwarp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int w = (cwarp >> 2) & 1;
    const int row = tid & 127;
    const uint32_t lane_sel = static_cast<uint32_t>((cwarp & 3) * 32) << 16;
    const uint32_t tS = tS_ + lane_sel + w * 64;
    const uint32_t tDP = tDP_ + lane_sel + w * 64;
    bool ok = true;
    int g0 = 0;
    uint32_t k = 0;
    // Row statistics of the next tile (rows r8 and r8 + 8 of the warp's block in the quad layout, else one row per thread), asked
    // for while the tile before is worked on; those of a block's first tile before the epilogue of the block before.
    float lse_nx[Cfg::kQuad ? 2 : 1], d_nx[Cfg::kQuad ? 2 : 1];
    int32_t bs_nx = 0;
    bool fetched = false;
    auto fetch_stats = [&](const BlockInfo& x, int t, uint32_t k) {
      if (ONE_LAUNCH) ok = mbar_wait_warp(smem_u32(&sh.stat_ready), 0, abort_flag);
      const int64_t stats = (static_cast<int64_t>(x.b) * ka.heads + x.h) * ka.lse_stride;  // row of LSE and D
      const int i0 = q_tile(x, t, k) * kBM + (Cfg::kQuad ? (cwarp & 3) * 32 + (cwarp >> 3) * 16 : row);
#pragma unroll
      for (int u = 0; u < (Cfg::kQuad ? 2 : 1); ++u) {
        const int i = Cfg::kQuad ? i0 + u * 8 + ((tid & 31) >> 2) : i0;
        const bool valid = i < x.sq;
        lse_nx[u] = valid ? ka.lse[stats + i] : INFINITY;  // scaled at its first use, one tile later
        d_nx[u] = valid ? a.softmax_d[stats + i] : 0.f;
      }
      if constexpr (BLOCKSPARSE)
        bs_nx = (i0 >> 4) < ka.bs_rows16
                    ? ka.bs_iter[(static_cast<int64_t>(x.b) * ka.bs_kblocks + (x.n0 >> 8)) * ka.bs_rows16 + (i0 >> 4)]
                    : -1;
    };
    // The warp's rows of the P~ and dS tiles are free for the first P~ of a block once the stores of the epilogue before
    // (by lane 0) have read them.
    auto rows_free = [&](int t) {
      if (!kTmaRows || t > 0 || k == 0) return;
      if ((tid & 31) == 0) bulk_wait_read();
      __syncwarp();
    };
    do {
    // with eight compute warps read where it is used, to hold few registers across the tiles (with sixteen, which have
    // them, 8 x 12 x 4096 with blocks taken over takes 973 us so and 924 from registers)
    using Block = std::conditional_t<Cfg::kQuad, const BlockInfo, const BlockInfo&>;
    Block x = sh.blk[k & 1];
    const int nm = x.nm;
    if (nm <= 0) {
      zero_tile(x, 32 * Cfg::kComputeWarps);
      continue;
    }
    const int64_t bh_sub =
        (static_cast<int64_t>(x.b) * ka.drop.heads_total + ka.drop.head_offset + x.h) * 256;
    if (!fetched) fetch_stats(x, 0, k);
    fetched = false;
    const uint64_t c2 = pack_f2(ka.scale_log2, ka.scale_log2);
    // dropout: per-lane generator state (lanes l and l ^ 8 share every Philox call)
    LanePhilox lp;
    float thr_term = 0.f;
    if constexpr (DROPOUT) {
      lp.init(ka.drop, bh_sub, row);
      thr_term = fa_keep_thr_term(ka.drop.threshold);
    }
    if constexpr (Cfg::kQuad) {
      // ---- d = 64 with dropout: quad layout.  A warp owns a 16-row block (hh) of its 32 lanes and one half of
      // the keys, and reads both products with the 16x256b shape: a thread holds rows r8 and r8 + 8 and
      // two adjacent columns of every 8-column unit, which is the ownership pattern of the reference's mask
      // generator (one Philox call = one thread's part of a 16 x 16 patch, QuadPhilox).  The packed
      // pairs go to the swizzled P~ / dS tiles with stmatrix (8 x 8 matrices = 16-byte row chunks).
      const int wq = cwarp & 3, hh = cwarp >> 3, lane = tid & 31;
      const int r8 = lane >> 2, q4 = lane & 3;
      const uint32_t tSq = tS + (static_cast<uint32_t>(hh * 16) << 16), tDPq = tDP + (static_cast<uint32_t>(hh * 16) << 16);
      QuadPhilox<4> qp;
      qp.init(ka.drop, bh_sub, lane, w * 4);
      // stmatrix row address of this lane: matrix k = lane / 8 is (row half k & 1, unit k >> 1)
      const int st_row = wq * 32 + hh * 16 + ((lane >> 3) & 1) * 8 + (lane & 7);
      const uint32_t st_off = w * 16384 + st_row * 128;
      const int st_unit = (lane >> 4) ^ (st_row & 7);  // unit 0 or 1 of a pair, swizzled (pairs start at even units)
      auto arrive_warp = [&](uint64_t& bar) {
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar));
      };
      for (int t = 0; t < nm && ok; ++t) {
        const int g = g0 + t;
        const int n0 = x.n0, sk = x.sk, L16 = (x.sq + 15) >> 4;
        const int cbase = n0 + w * 64;  // first key column of this thread
        const int m0 = q_tile(x, t, k) * kBM;
        const int row0 = m0 + wq * 32 + hh * 16 + r8;  // + 8 * u
        uint64_t nlse2[2], nd2[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float l2 = lse_nx[u] * 1.4426950408889634f;
          nlse2[u] = pack_f2(-l2, -l2);
          nd2[u] = pack_f2(-d_nx[u], -d_nx[u]);
        }
        const int32_t bs_it = bs_nx;
        if (t + 1 < nm) fetch_stats(x, t + 1, k);
        // (a block that is not in the layout is masked too)
        const bool need_mask = (n0 + kBN > sk) || (CAUSAL && (n0 + kBN - 1 > m0)) || (BLOCKSPARSE && bs_it < 0);

        // keep words of the thread's four patches (they do not depend on the scores: drawn before the wait).
        // kw[grp][2 * u + half]: row u, columns 16 grp + 8 half + 2 q4 (+1 in the high 16 bits)
        uint32_t kw[4][4];
        {
          int64_t it_tile;
          if constexpr (BLOCKSPARSE) it_tile = bs_it;
          else it_tile = fa_iter_index(CAUSAL, n0 >> ka.drop.n_shift, (m0 + wq * 32 + hh * 16) >> 4, L16, ka.drop.n_shift);
          qp.set_tile(ka.drop, it_tile, n0);
#pragma unroll
          for (int g4 = 0; g4 < 4; ++g4) qp.start(g4, kw[g4]);
#pragma unroll
          for (int r = 2; r < 7; ++r)
#pragma unroll
            for (int g4 = 0; g4 < 4; ++g4) QuadPhilox<4>::round(ka.drop, kw[g4], r);
        }
        ok = mbar_wait_warp<kVote>(smem_u32(&sh.sdp_full), g & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        // 32 columns after the other: 16 scores, 16 dP values a thread
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t sr[16], dr[16];  // [4 * unit + 2 * u + column]
          tmem_ld_quad16(tSq + c * 32, sr);
          tmem_ld_quad16(tDPq + c * 32, dr);
          tmem_wait_ld();
          if (c == 1) {
            tc_fence_before();
            arrive_warp(sh.sdp_consumed);
          }
          uint32_t pp[8], pds[8];  // [2 * unit + u]: the stmatrix register order
          auto block_math = [&](auto masked) {
#pragma unroll
            for (int unit = 0; unit < 4; ++unit) {
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int i = 4 * unit + 2 * u;
                float p0, p1;
                unpack_f2(fma2(pack_f2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), c2, nlse2[u]), p0, p1);
                p0 = ex2f(p0);
                p1 = ex2f(p1);
                if constexpr (decltype(masked)::value) {
                  const int col = cbase + c * 32 + unit * 8 + 2 * q4, ig = row0 + u * 8;
                  bool v0 = col < sk, v1 = col + 1 < sk;
                  if (CAUSAL) { v0 = v0 && (col <= ig); v1 = v1 && (col + 1 <= ig); }
                  if (BLOCKSPARSE && bs_it < 0) { v0 = false; v1 = false; }
                  if (!v0) p0 = 0.f;
                  if (!v1) p1 = 0.f;
                }
                const uint32_t word = kw[2 * c + (unit >> 1)][2 * u + (unit & 1)];
                const uint64_t p01 = pack_f2(p0, p1);
                const uint64_t k01 = mul2(p01, pack_f2(fa_keep_factor_lo(word, thr_term), fa_keep_factor_hi(word, thr_term)));
                float k0, k1, s0, s1;
                unpack_f2(k01, k0, k1);
                // dS = P~ * dP - P * D  (P~ = P where kept, 0 where dropped)
                unpack_f2(fma2(k01, pack_f2(__uint_as_float(dr[i]), __uint_as_float(dr[i + 1])), mul2(p01, nd2[u])), s0, s1);
                pp[2 * unit + u] = pack_lowp<BF16>(k0, k1);
                pds[2 * unit + u] = pack_lowp<BF16>(s0, s1);
              }
            }
          };
          if (need_mask) block_math(std::true_type{}); else block_math(std::false_type{});
          // the previous tile's products must have finished reading the P~ / dS buffers
          if (c == 0 && g > 0) {
            ok = mbar_wait_warp<kVote>(smem_u32(&sh.pds_free), (g & 1) ^ 1, abort_flag);
            if (!ok) break;
            rows_free(t);
          }
          // four 8 x 8 matrices per instruction: (u = 0, 1) x (units a, a + 1) of the 64-column panel w
#pragma unroll
          for (int a2 = 0; a2 < 4; a2 += 2) {
            const uint32_t off = st_off + (((c * 4 + a2) ^ st_unit) << 4);
            stmatrix_x4(smem_u32(p_ptr) + off, pp[2 * a2], pp[2 * a2 + 1], pp[2 * a2 + 2], pp[2 * a2 + 3]);
            stmatrix_x4(smem_u32(ds_ptr) + off, pds[2 * a2], pds[2 * a2 + 1], pds[2 * a2 + 2], pds[2 * a2 + 3]);
          }
        }
        if (!ok) break;
        fence_async_smem();
        arrive_warp(sh.pds_ready);
      }
    } else {

    for (int t = 0; t < nm && ok; ++t) {
      const int g = g0 + t;
      const int n0 = x.n0, sk = x.sk, L16 = (x.sq + 15) >> 4;
      const int cbase = n0 + w * 64;  // first key column of this thread
      const int m0 = q_tile(x, t, k) * kBM;
      const int ig = m0 + row;
      const float lse2 = lse_nx[0] * 1.4426950408889634f;
      const float d_i = d_nx[0];
      const uint64_t nlse2 = pack_f2(-lse2, -lse2);
      const uint64_t nd2 = pack_f2(-d_i, -d_i);
      const int32_t bs_it = bs_nx;
      const bool row_in_layout = !BLOCKSPARSE || bs_it >= 0;
      if (t + 1 < nm) fetch_stats(x, t + 1, k);

      // Keep words of this thread's 64 columns (wd[p] covers columns 2p, 2p + 1).  They do not depend
      // on the scores, so they are drawn before the wait for S and dP: eight independent Philox
      // calls (4 column groups x 2 quarters) with their rounds interleaved.
      uint32_t wd[DROPOUT ? 32 : 1];
      if constexpr (DROPOUT) {
        // one Philox iteration index per tile: a 128-column tile lies inside one key block
        int64_t it_tile;
        if constexpr (BLOCKSPARSE) it_tile = bs_it;
        else it_tile = fa_iter_index(CAUSAL, n0 >> ka.drop.n_shift, ig >> 4, L16, ka.drop.n_shift);
        lp.set_tile(ka.drop, it_tile, n0);
        uint32_t st[8][4];
#pragma unroll
        for (int g4 = 0; g4 < 4; ++g4) {
          lp.start(w * 4 + g4, 0, st[2 * g4]);
          lp.start(w * 4 + g4, 1, st[2 * g4 + 1]);
        }
#pragma unroll
        for (int r = 0; r < 7; ++r)
#pragma unroll
          for (int k8 = 0; k8 < 8; ++k8) lp.round(st[k8], r);
#pragma unroll
        for (int g4 = 0; g4 < 4; ++g4) lp.finish(st[2 * g4], st[2 * g4 + 1], wd + g4 * 8);
      }

      // one decision for the warp: its threads' rows may lie in two 16-row blocks of the layout
      const bool need_mask = (n0 + kBN > sk) || (CAUSAL && (n0 + kBN - 1 > m0)) ||
                             (BLOCKSPARSE && __any_sync(0xffffffffu, !row_in_layout));
      if constexpr (Cfg::kTwoPhase) {
        // ---- phase one: P from S.  P~ goes to shared memory (dV can start), P stays in registers.
        ok = mbar_wait(smem_u32(&sh.s_full), g & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        uint32_t pf[2][32];
        auto phase_one = [&](auto masked) {
        constexpr bool kMasked = decltype(masked)::value;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t sr[32];
          tmem_ld32(tS + c * 32, sr);
          tmem_wait_ld();
          if (c == 1) {
            tc_fence_before();
            mbar_arrive(smem_u32(&sh.sdp_consumed));
          }
          uint32_t pp[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float p0, p1;
            unpack_f2(fma2(pack_f2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), c2, nlse2), p0, p1);
            p0 = ex2f(p0);
            p1 = ex2f(p1);
            if (kMasked && need_mask) {
              const int col = cbase + c * 32 + i;
              bool v0 = col < sk, v1 = col + 1 < sk;
              if (CAUSAL) { v0 = v0 && (col <= ig); v1 = v1 && (col + 1 <= ig); }
              if (BLOCKSPARSE && !row_in_layout) { v0 = false; v1 = false; }
              if (!v0) p0 = 0.f;
              if (!v1) p1 = 0.f;
            }
            pf[c][i] = __float_as_uint(p0);
            pf[c][i + 1] = __float_as_uint(p1);
            float k0 = p0, k1 = p1;
            if constexpr (DROPOUT) {
              const uint32_t word = wd[c * 16 + (i >> 1)];
              unpack_f2(mul2(pack_f2(p0, p1),
                             pack_f2(fa_keep_factor_lo(word, thr_term), fa_keep_factor_hi(word, thr_term))), k0, k1);
            }
            pp[i >> 1] = pack_lowp<BF16>(k0, k1);
          }
          // dV of the previous tile must have finished reading the P~ buffer
          if (c == 0 && g > 0) {
            ok = mbar_wait(smem_u32(&sh.pds_free), (g & 1) ^ 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            rows_free(t);
          }
#pragma unroll
          for (int ch4 = 0; ch4 < 4; ++ch4) {
            const int ch = c * 4 + ch4;
            const uint32_t off = w * 16384 + row * 128 + ((ch ^ (row & 7)) << 4);
            *reinterpret_cast<uint4*>(p_ptr + off) =
                make_uint4(pp[4 * ch4], pp[4 * ch4 + 1], pp[4 * ch4 + 2], pp[4 * ch4 + 3]);
          }
        }
        };
        if (need_mask) phase_one(std::true_type{}); else phase_one(std::false_type{});
        if (!ok) break;
        fence_async_smem();
        mbar_arrive(smem_u32(&sh.p_ready));

        // ---- phase two: dS = P~ * dP - P * D from dP
        ok = mbar_wait(smem_u32(&sh.sdp_full), g & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t dr[32];
          tmem_ld32(tDP + c * 32, dr);
          tmem_wait_ld();
          uint32_t pds[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const uint64_t p01 = pack_f2(__uint_as_float(pf[c][i]), __uint_as_float(pf[c][i + 1]));
            uint64_t k01 = p01;
            if constexpr (DROPOUT) {
              const uint32_t word = wd[c * 16 + (i >> 1)];
              k01 = mul2(p01, pack_f2(fa_keep_factor_lo(word, thr_term), fa_keep_factor_hi(word, thr_term)));
            }
            float s0, s1;
            unpack_f2(fma2(k01, pack_f2(__uint_as_float(dr[i]), __uint_as_float(dr[i + 1])), mul2(p01, nd2)), s0, s1);
            pds[i >> 1] = pack_lowp<BF16>(s0, s1);
          }
          // dK, dQ of the previous tile must have finished reading the dS buffer
          if (c == 0 && g > 0) {
            ok = mbar_wait(smem_u32(&sh.ds_free), (g & 1) ^ 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
          }
#pragma unroll
          for (int ch4 = 0; ch4 < 4; ++ch4) {
            const int ch = c * 4 + ch4;
            const uint32_t off = w * 16384 + row * 128 + ((ch ^ (row & 7)) << 4);
            *reinterpret_cast<uint4*>(ds_ptr + off) =
                make_uint4(pds[4 * ch4], pds[4 * ch4 + 1], pds[4 * ch4 + 2], pds[4 * ch4 + 3]);
          }
          // second copy of dS for the dQ product, over this group's own scores, which every thread of it has read
          if constexpr (kDsInTmem) tmem_st16(tDS_ + lane_sel + w * 64 + c * 16, pds);
        }
        tc_fence_before();  // the dP columns are about to be overwritten by dQ
      } else {
      ok = mbar_wait(smem_u32(&sh.sdp_full), g & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();

      // d = 64 without dropout.  This thread's 64 scores and 64 dP values go to registers at once, so that the next
      // tile's S and dP products can overwrite tensor memory while this tile is still being processed.
      uint32_t sr[2][32], dr[2][32];
      tmem_ld32(tS, sr[0]);
      tmem_ld32(tS + 32, sr[1]);
      tmem_ld32(tDP, dr[0]);
      tmem_ld32(tDP + 32, dr[1]);
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive(smem_u32(&sh.sdp_consumed));
      auto tile_math = [&](auto masked) {
      constexpr bool kMasked = decltype(masked)::value;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pp[16], pds[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float p0, p1;
          unpack_f2(fma2(pack_f2(__uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1])), c2, nlse2), p0, p1);
          p0 = ex2f(p0);
          p1 = ex2f(p1);
          if constexpr (kMasked) {
            const int col = cbase + c * 32 + i;
            bool v0 = col < sk, v1 = col + 1 < sk;
            if (CAUSAL) { v0 = v0 && (col <= ig); v1 = v1 && (col + 1 <= ig); }
            if (BLOCKSPARSE && !row_in_layout) { v0 = false; v1 = false; }
            if (!v0) p0 = 0.f;
            if (!v1) p1 = 0.f;
          }
          const uint64_t p01 = pack_f2(p0, p1);
          float s0, s1;  // dS = P * dP - P * D
          unpack_f2(fma2(p01, pack_f2(__uint_as_float(dr[c][i]), __uint_as_float(dr[c][i + 1])), mul2(p01, nd2)), s0, s1);
          pp[i >> 1] = pack_lowp<BF16>(p0, p1);
          pds[i >> 1] = pack_lowp<BF16>(s0, s1);
        }
        // the previous tile's products must have finished reading the P~ / dS buffers
        if (c == 0 && g > 0) {
          ok = mbar_wait(smem_u32(&sh.pds_free), (g & 1) ^ 1, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          rows_free(t);
        }
        // 32 16-bit values = 4 chunks of 16 bytes of this row in the 64-column panel w
#pragma unroll
        for (int ch4 = 0; ch4 < 4; ++ch4) {
          const int ch = c * 4 + ch4;
          const uint32_t off = w * 16384 + row * 128 + ((ch ^ (row & 7)) << 4);
          *reinterpret_cast<uint4*>(p_ptr + off) =
              make_uint4(pp[4 * ch4], pp[4 * ch4 + 1], pp[4 * ch4 + 2], pp[4 * ch4 + 3]);
          *reinterpret_cast<uint4*>(ds_ptr + off) =
              make_uint4(pds[4 * ch4], pds[4 * ch4 + 1], pds[4 * ch4 + 2], pds[4 * ch4 + 3]);
        }
        // second copy of dS for the dQ product (32 keys = 16 packed columns of this half)
        tmem_st16(tDS_ + lane_sel + w * 32 + c * 16, pds);
      }
      };
      if (need_mask) tile_math(std::true_type{}); else tile_math(std::false_type{});
      }
      if (!ok) break;
      if constexpr (kDsInTmem) {
        tmem_wait_st();
        tc_fence_before();
      }
      fence_async_smem();
      mbar_arrive(smem_u32(&sh.pds_ready));
    }
    }  // row-per-thread layout

    // ---------------- epilogue: group 0 writes dV = acc / p_keep, group 1 writes dK = acc * scale / p_keep
    if (ok && take_over) {
      ok = mbar_wait_warp<kVote>(smem_u32(&sh.blk_full[(k + 1) & 1]), (k >> 1) & 1, abort_flag);
      fetched = ok && sh.blk[(k + 1) & 1].nm > 0;
      if (fetched) fetch_stats(sh.blk[(k + 1) & 1], 0, k + 1);
    }
    if (ok) {
      ok = mbar_wait(smem_u32(&sh.pds_free), (g0 + nm - 1) & 1, abort_flag);
      if constexpr (Cfg::kTwoPhase) {
        if (ok) ok = mbar_wait(smem_u32(&sh.ds_free), (g0 + nm - 1) & 1, abort_flag);
      }
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after();
      // From tid (see `warp`): held from the start of the role instead, d = 128 with dropout and no causal mask takes 1437 us
      // for 4 x 12 x 4096, so 1352.
      const int grp = (tid >> 7) & 1;
      // sixteen warps: warps 8-15 take the second half of the columns
      const int part = Cfg::kQuad ? tid >> 8 : 0;
      constexpr int kChunks = Cfg::kQuad ? D / 64 : D / 32;
      const uint32_t tAcc = (grp == 0 ? tDV_ : tDK_) + (static_cast<uint32_t>(((tid >> 5) & 3) * 32) << 16);
      const float f = (grp == 0) ? rp_keep : ka.scale * rp_keep;
      const BlockInfo e = sh.blk[k & 1];
      const int r0 = e.n0 + ((tid >> 5) & 3) * 32;  // first key row of the warp
      const int64_t stride = grp == 0 ? a.dv_row_stride : a.dk_row_stride;
      uint16_t* dst = (grp == 0 ? dv_base : dk_base) + static_cast<int64_t>(e.k_start + r0) * stride +
                      static_cast<int64_t>(e.h) * (grp == 0 ? a.dv_head_stride : a.dk_head_stride) + part * (kChunks * 32);
      // Out through the rows of the P~ and dS tiles that this warp alone writes (see stage_offset): other warps may be in the
      // next block already.
      constexpr int CH = Cfg::kQuad ? 4 : 8;  // 16-byte chunks of a row that a warp holds at once
      static_assert(!kTmaRows || kBoxColumns == CH * 8, "box of tm_dk and tm_dv");
      const uint32_t piece = grp * 16384 + ((tid >> 5) & 3) * 4096 + part * 2048;
#pragma unroll
      for (int i = 0; i < kChunks; ++i) {
        uint32_t r[32];
        tmem_ld32(tAcc + (part * kChunks + i) * 32, r);
        tmem_wait_ld();
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint32_t pk[4];
#pragma unroll
          for (int k = 0; k < 4; ++k)
            pk[k] = pack_lowp<BF16>(__uint_as_float(r[8 * v + 2 * k]) * f, __uint_as_float(r[8 * v + 2 * k + 1]) * f);
          *reinterpret_cast<uint4*>((i / 2 == 0 ? p_ptr : ds_ptr) + piece + stage_offset<CH>(tid & 31, (i & 1) * 4 + v)) =
              make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
      }
      tc_fence_before();
      fence_async_smem();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(smem_u32(&sh.acc_free));
      // Whole rows by TMA, which leaves the warp free for the next block (64 KB through the LSU took it 3500 clk at d = 128, with
      // the first statistics of the next block behind them another 2350; a query tile takes 5500).  The warp that holds the
      // sequence's end stores its rows itself, since those behind it are the next sequence's.
      if (kTmaRows && r0 + 32 <= e.sk) {
        if ((tid & 31) == 0) {
#pragma unroll
          for (int p = 0; p < (kChunks + 1) / 2; ++p)
            if (part * 32 + p * 64 < ka.head_dim)
              tma_store_3d(grp == 0 ? &tm_dv : &tm_dk, smem_u32(p == 0 ? p_ptr : ds_ptr) + piece,
                           part * 32 + p * 64, e.k_start + r0, e.h);
          bulk_commit();
        }
      } else {
#pragma unroll
        for (int p = 0; p < (kChunks + 1) / 2; ++p)
          stage_copy_out<CH>((p == 0 ? p_ptr : ds_ptr) + piece, dst + p * 64, stride, e.sk - r0,
                             ka.head_dim / 8 - part * 4 - p * 8, tid & 31);
      }
    }
    g0 += nm;
    } while (ok && next_block(k++));
    if ((tid & 31) == 0) bulk_wait_all();
  } else {
    // ------------------------------------------------------------------ dQ group
    // dQ tile: tensor memory -> registers -> swizzled fp32 staging in shared memory -> one TMA
    // reduce-add per [128 rows x 32 columns] box into the fp32 accumulator.  Rows past the end of
    // the sequence hold exact zeros (their P is zero), rows past the tensor are clipped by TMA.
    reg_dealloc<Cfg::kDqRegs>();
    grid_dep_wait();
    const int row = tid - 32 * kDqWarp;
    const uint32_t lane_sel = static_cast<uint32_t>((__shfl_sync(0xffffffffu, tid >> 5, 0) & 3) * 32) << 16;
    const uint32_t tDQ = tDQ_ + lane_sel;
    const uint32_t stage_addr = smem_u32(dq_stage);
    bool ok = true;
    bool pending = false;  // thread `row == 0`: a reduce group of this CTA may still read the staging
    uint32_t sync_phase = 0;
    auto group_sync = [&]() -> bool {
      mbar_arrive(smem_u32(&sh.dq_group));
      const bool done = mbar_wait(smem_u32(&sh.dq_group), sync_phase & 1, abort_flag);
      ++sync_phase;
      return done;
    };
    // Deterministic mode (thread `row == 0` only): wait until the key tiles before this one have
    // added their share of the query tile, add, wait for the adds to complete and pass the turn on.
    // (no blocks are taken over: one row of tickets)
    int32_t* const ticket_row =
        deterministic ? a.dq_tickets + (static_cast<int64_t>(first.b) * ka.heads + first.h) * a.ticket_stride : nullptr;
    auto ticket_wait = [&](const BlockInfo& x, int t, int m) -> bool {
      int32_t want;
      if constexpr (BLOCKSPARSE) want = qtile_order[t];
      else want = x.n0 / kBN;
      const volatile int32_t* tk = ticket_row + m;
      if (*abort_flag) return false;
      const long long t0 = clock64();
      while (true) {
        int32_t cur;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(cur) : "l"(tk) : "memory");
        if (cur >= want) break;
        if (*abort_flag) return false;
        if (clock64() - t0 > WAIT_LIMIT_CYCLES) { *abort_flag = 1; return false; }
      }
      // the adds below go through the async proxy
      asm volatile("fence.proxy.async.global;" ::: "memory");
      return true;
    };
    bool my_turn = true;
    auto ticket_pass = [&](int m) {
      bulk_wait_all();
      asm volatile("fence.proxy.async.global;" ::: "memory");
      __threadfence();
      int32_t* tk = ticket_row + m;
      asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(tk) : "memory");
    };
    // One launch: softmax_d = p_keep * rowsum(dO * O), 32 rows a warp, in the order of bwd_preprocess_kernel.
    auto write_d = [&](const BlockInfo& x) {
      const int dlane = row & 31, tpr = ka.head_dim / 8, rows = 32 / tpr;
      const int r0 = (row & ~31) + dlane / tpr;
      const int64_t token = x.q_start + r0;
      const uint16_t* o = reinterpret_cast<const uint16_t*>(a.o_in) + token * ka.o_row_stride + x.h * ka.o_head_stride + (dlane % tpr) * 8;
      const uint16_t* dout = reinterpret_cast<const uint16_t*>(a.dout) + token * a.do_row_stride + x.h * a.do_head_stride + (dlane % tpr) * 8;
      float* d = a.softmax_d + (static_cast<int64_t>(x.b) * ka.heads + x.h) * ka.lse_stride + r0;
#pragma unroll 4
      for (int i = 0; i < tpr; ++i) {
        const bool valid = r0 + i * rows < x.sq;
        float acc = 0.f;
        if (valid)
          acc = dot8<BF16>(*reinterpret_cast<const uint4*>(o + i * rows * ka.o_row_stride),
                           *reinterpret_cast<const uint4*>(dout + i * rows * a.do_row_stride));
        for (int off = tpr / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
        if (valid && dlane % tpr == 0) d[i * rows] = acc * a.p_keep;
      }
      __syncwarp();
      if (dlane == 0) mbar_arrive(smem_u32(&sh.stat_ready));
    };
    // One launch: this warp's 32 rows of a dQ tile are all of dQ.
    auto write_dq = [&](const BlockInfo& x) {
      const int dlane = row & 31, r0 = row & ~31;
      const float f = ka.scale * ka.rp_keep;
      uint8_t* piece = dq_stage + (row >> 5) * 4096;
      uint16_t* dst = reinterpret_cast<uint16_t*>(a.dq) + (x.q_start + r0) * a.dq_row_stride + x.h * a.dq_head_stride;
#pragma unroll 1
      for (int half = 0; half < D / 64; ++half) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t r[16];
          tmem_ld16(tDQ + half * 64 + c * 16, r);
          tmem_wait_ld();
          uint32_t pk[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            pk[i] = x.sk > 0 ? pack_lowp<BF16>(__uint_as_float(r[2 * i]) * f, __uint_as_float(r[2 * i + 1]) * f) : 0;
          *reinterpret_cast<uint4*>(piece + stage_offset<8>(dlane, 2 * c)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          *reinterpret_cast<uint4*>(piece + stage_offset<8>(dlane, 2 * c + 1)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
        __syncwarp();
        stage_copy_out<8>(piece, dst + half * 64, a.dq_row_stride, x.sq - r0, ka.head_dim / 8 - half * 8, dlane);
        __syncwarp();
      }
    };
    int g = 0;
    uint32_t k = 0;
    do {
    const BlockInfo& x = sh.blk[k & 1];  // read where it is used: the group has few registers
    const int nm = x.nm;
    if constexpr (ONE_LAUNCH) {
      if (nm <= 0) continue;
      write_d(x);
      ok = mbar_wait_warp(smem_u32(&sh.dq_full), 0, abort_flag);
      if (ok) {
        tc_fence_after();
        write_dq(x);
      }
    } else {
    for (int t = 0; t < nm && ok; ++t, ++g) {
      const int m = q_tile(x, t, k), q_row = x.q_start + m * kBM, q_head = x.h;  // ahead of the waits
      ok = mbar_wait(smem_u32(&sh.dq_full), g & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      if constexpr (Cfg::kAliasDq) {
        // dQ shares its columns with the next dP, so the columns are released as early as possible:
        // both boxes of a 64-column half go to registers before anything waits for the staging
        // buffer, and the release follows the loads of the second half.
#pragma unroll
        for (int half = 0; half < D / 64; ++half) {
          uint32_t r0[32], r1[32];
          tmem_ld32(tDQ + half * 64, r0);
          tmem_ld32(tDQ + half * 64 + 32, r1);
          tmem_wait_ld();
          if (half == D / 64 - 1) {
            tc_fence_before();
            mbar_arrive(smem_u32(&sh.dq_consumed));
          }
          // the staging buffer is free once the previous reduce has read it
          if (row == 0 && pending) bulk_wait_read();
          ok = group_sync();
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
#pragma unroll
          for (int ch = 0; ch < 8; ++ch) {
            const uint32_t off = row * 128 + ((ch ^ (row & 7)) << 4);
            *reinterpret_cast<uint4*>(dq_stage + off) = make_uint4(r0[4 * ch], r0[4 * ch + 1], r0[4 * ch + 2], r0[4 * ch + 3]);
            *reinterpret_cast<uint4*>(dq_stage + 16384 + off) = make_uint4(r1[4 * ch], r1[4 * ch + 1], r1[4 * ch + 2], r1[4 * ch + 3]);
          }
          fence_async_smem();
          ok = group_sync();
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          if (row == 0) {
            // on expiry the abort flag is set, this tile's add is skipped and every role leaves
            // at its next wait
            if (deterministic && half == 0) my_turn = ticket_wait(x, t, m);
            if (my_turn) {
              tma_reduce_add_3d(&tm_dq, stage_addr, half * 64, q_row, q_head);
              tma_reduce_add_3d(&tm_dq, stage_addr + 16384, half * 64 + 32, q_row, q_head);
              bulk_commit();
              pending = true;
              if (deterministic && half == D / 64 - 1) { ticket_pass(m); pending = false; }
            }
          }
        }

      } else {
#pragma unroll
      for (int half = 0; half < D / 64; ++half) {
#pragma unroll
        for (int bx = 0; bx < 2; ++bx) {
          uint32_t r[32];
          tmem_ld32(tDQ + half * 64 + bx * 32, r);
          tmem_wait_ld();
          if (half == D / 64 - 1 && bx == 1) {
            tc_fence_before();
            mbar_arrive(smem_u32(&sh.dq_consumed));
          }
          if (bx == 0) {
            // the staging buffer is free once the previous reduce has read it
            if (row == 0 && pending) bulk_wait_read();
            ok = group_sync();
            ok = __all_sync(0xffffffffu, ok);
          }
          if (ok) {
#pragma unroll
            for (int ch = 0; ch < 8; ++ch) {
              const uint32_t off = bx * 16384 + row * 128 + ((ch ^ (row & 7)) << 4);
              *reinterpret_cast<uint4*>(dq_stage + off) = make_uint4(r[4 * ch], r[4 * ch + 1], r[4 * ch + 2], r[4 * ch + 3]);
            }
          }
        }
        if (!ok) break;
        fence_async_smem();
        ok = group_sync();
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (row == 0) {
          if (deterministic && half == 0) my_turn = ticket_wait(x, t, m);
          if (my_turn) {
            tma_reduce_add_3d(&tm_dq, stage_addr, half * 64, q_row, q_head);
            tma_reduce_add_3d(&tm_dq, stage_addr + 16384, half * 64 + 32, q_row, q_head);
            bulk_commit();
            pending = true;
            if (deterministic && half == D / 64 - 1) { ticket_pass(m); pending = false; }
          }
        }
      }
      }
    }
    }
    } while (ok && next_block(k++));
    if (row == 0 && pending) bulk_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kProducer) {
    tmem_dealloc(tmem, 512);
    if (lane == 0 && sh.abort_flag && ka.status) {
      atomicExch(ka.status, ka.launch_id);  // stops the CTAs of this launch that have not started yet
      atomicExch(ka.status + 3, 1);  // sticky: read by the host
    }
  }
}

// ------------------------------------------------------------------------------------------------
// softmax_d = p_keep * rowsum(dO * O); zero the dQ accumulator.  One thread per 8 elements.
template <bool BF16>
__global__ void bwd_preprocess_kernel(const BwdArgs a, int dpad) {
  grid_dep_wait();
  const KernelArgs& ka = a.k;
  const int b = blockIdx.z, h = blockIdx.y;
  const int q_start = ka.cu_seqlens_q[b];
  const int sq = ka.cu_seqlens_q[b + 1] - q_start;
  const int d = ka.head_dim;
  const int tpr = d / 8;                      // threads per row: 2, 4, 8 or 16
  const int rows_per_block = blockDim.x / tpr;
  const int r = threadIdx.x / tpr, c = (threadIdx.x % tpr) * 8;
  const int i = blockIdx.x * rows_per_block + r;
  if (a.dq_tickets != nullptr && blockIdx.x == 0) {
    int32_t* tk = a.dq_tickets + (static_cast<int64_t>(b) * ka.heads + h) * a.ticket_stride;
    for (int t = threadIdx.x; t < a.ticket_stride; t += blockDim.x) tk[t] = 0;
  }
  // A block behind its sequence's last row, of which uneven batches have many, ends without the signal, which its end stands for:
  // two sequences of 16384 and 126 of 64 tokens, 4 heads, this kernel 553 -> 293 us (d = 128; 398 without the two instructions).
  if (static_cast<int>(blockIdx.x) * rows_per_block >= sq) return;
  // (behind the wait: the main kernel's first loads rely on everything ahead of this kernel being over)
  grid_dep_launch();
  float acc = 0.f;
  if (i < sq) {
    const int64_t row = q_start + i;
    const uint16_t* o = reinterpret_cast<const uint16_t*>(a.o_in) + row * ka.o_row_stride + h * ka.o_head_stride + c;
    const uint16_t* g = reinterpret_cast<const uint16_t*>(a.dout) + row * a.do_row_stride + h * a.do_head_stride + c;
    // (O, like the accumulator below, is not read again: what is leaves more of the accumulator in the L2.  Whole backward, us:
    // 16 x 12 x 1000 causal (d = 128) 253 -> 250, 32 x 12 x 512 185 -> 183)
    const uint4 ov = __ldcs(reinterpret_cast<const uint4*>(o));
    const uint4 gv = *reinterpret_cast<const uint4*>(g);
    acc = dot8<BF16>(ov, gv);
    // zero this thread's share of the fp32 dQ accumulator row (dpad floats per (row, head))
    float* zr = a.dq_accum + (row * ka.heads + h) * dpad;
    for (int z = (threadIdx.x % tpr) * 4; z < dpad; z += tpr * 4)
      *reinterpret_cast<float4*>(zr + z) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int off = tpr / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (i < sq && (threadIdx.x % tpr) == 0)
    a.softmax_d[(static_cast<int64_t>(b) * ka.heads + h) * ka.lse_stride + i] = acc * a.p_keep;
}

// dq = accumulator * scale / p_keep.  One thread per 8 elements.
template <bool BF16>
__global__ void bwd_postprocess_kernel(const BwdArgs a, int dpad) {
  grid_dep_wait();
  const KernelArgs& ka = a.k;
  const int d = ka.head_dim;
  const int tpr = d / 8;
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t total = static_cast<int64_t>(a.total_q) * ka.heads * tpr;
  if (idx >= total) return;
  const int c = static_cast<int>(idx % tpr) * 8;
  const int64_t rh = idx / tpr;
  const int h = static_cast<int>(rh % ka.heads);
  const int64_t row = rh / ka.heads;
  // Rows behind the last sequence (a token buffer larger than cu_seqlens_q[batch]) belong to nobody:
  // the accumulator was not cleared there and dq keeps what the caller put in it, as in the
  // reference, which only ever writes rows of a sequence.
  if (row >= ka.cu_seqlens_q[ka.batch]) return;
  const float* src = a.dq_accum + rh * dpad + c;
  const float4 x = __ldcs(reinterpret_cast<const float4*>(src));
  const float4 y = __ldcs(reinterpret_cast<const float4*>(src + 4));
  const float f = ka.scale * ka.rp_keep;
  uint4 out;
  out.x = pack16<BF16>(x.x * f, x.y * f);
  out.y = pack16<BF16>(x.z * f, x.w * f);
  out.z = pack16<BF16>(y.x * f, y.y * f);
  out.w = pack16<BF16>(y.z * f, y.w * f);
  uint16_t* dst = reinterpret_cast<uint16_t*>(a.dq) + row * a.dq_row_stride + h * a.dq_head_stride + c;
  *reinterpret_cast<uint4*>(dst) = out;
}

template <int D, bool BF16, bool CAUSAL, bool DROPOUT, bool BS, bool ONE_LAUNCH = false, bool SHORT = false>
cudaError_t launch_main(const BwdLaunch& l, cudaStream_t stream) {
  if constexpr (!BS && !ONE_LAUNCH && !SHORT) {
    if (l.args.one_launch) return launch_main<D, BF16, CAUSAL, DROPOUT, BS, true>(l, stream);
    if constexpr (D == 64)
      if (short_queries(l)) return launch_main<D, BF16, CAUSAL, DROPOUT, BS, false, true>(l, stream);
  }
  auto kernel = fa_bwd_kernel<D, BF16, CAUSAL, DROPOUT, BS, ONE_LAUNCH, SHORT>;
  using Cfg = BwdCfg<D, BS, DROPOUT, SHORT>;
  constexpr int smem = Cfg::kSmemBytes;
  static SmemLimitFlags smem_limit_set;  // one per template instantiation of this function
  cudaError_t e = set_smem_limit_once(kernel, smem, smem_limit_set);
  if (e != cudaSuccess) return e;
  dim3 grid((l.args.max_seqlen_k + kBN - 1) / kBN, l.args.k.heads, l.args.k.batch);
  BwdArgs args = l.args;
  // Up to an SM per block all blocks start at once: no order, no block to take over, and the place of a block without divisions
  // (causal, us: 4 x 4 x 600 ragged 28.8 -> 28.3 at d = 128, 12 x 12 x 128 16.1 -> 16.0 at d = 64).
  const bool linear = linear_grid(grid.x, grid.y, grid.z) && int64_t(grid.x) * grid.y * grid.z > kSms;
  args.k.grid_tiles = grid.x;
  args.take_over = linear && l.args.dq_tickets == nullptr;
  if constexpr (CAUSAL) set_causal_grid(&args.k, grid.x, int64_t(8) * D * args.max_seqlen_q);  // Q, dO and the fp32 dQ
  if (linear && (CAUSAL || args.take_over)) grid = dim3(grid.x * grid.y * grid.z, 1, 1);
  // (not the main kernel of d = 128, causal, with dropout: its grid is slower when it starts beside the preprocess.  Whole backward
  // over its time with ordinary launches, all three overlapped -> now: 16 x 12 x 1000 1.024 -> 1.003, 4 x 12 x 4096 1.015 -> 1.000,
  // 4 x 12 x 1024 1.033 -> 0.985, 8 x 12 x 512 1.028 -> 0.973.)
  constexpr bool kOverlap = !(D == 128 && CAUSAL && DROPOUT);
  return launch(kOverlap && overlap_launches(l), kernel, grid, Cfg::kThreads, smem, stream, l.tm_q, l.tm_k, l.tm_v, l.tm_do, l.tm_dq, l.tm_dk, l.tm_dv, args);
}

template <int D, bool BF16, bool CAUSAL>
cudaError_t launch_dd(const BwdLaunch& l, cudaStream_t stream) {
  return l.is_dropout ? launch_main<D, BF16, CAUSAL, true, false>(l, stream)
                      : launch_main<D, BF16, CAUSAL, false, false>(l, stream);
}

template <int D>
cudaError_t launch_d(const BwdLaunch& l, cudaStream_t stream) {
  if (l.is_bf16) {
    return l.is_causal ? launch_dd<D, true, true>(l, stream) : launch_dd<D, true, false>(l, stream);
  }
  return l.is_causal ? launch_dd<D, false, true>(l, stream) : launch_dd<D, false, false>(l, stream);
}

}  // namespace

cudaError_t launch_bwd(const BwdLaunch& l, cudaStream_t stream) {
  const BwdArgs& a = l.args;
  const int d = a.k.head_dim;
  const int stages = l.stage_mask == 0 ? 7 : l.stage_mask;
  // 1. preprocess
  if ((stages & 1) && !a.one_launch) {
    const int tpr = d / 8;
    const int threads = 256;
    const int rows_per_block = threads / tpr;
    dim3 grid((a.max_seqlen_q + rows_per_block - 1) / rows_per_block, a.k.heads, a.k.batch);
    cudaError_t e = launch(overlap_launches(l), l.is_bf16 ? bwd_preprocess_kernel<true> : bwd_preprocess_kernel<false>, grid,
                           threads, 0, stream, a, l.dpad);
    if (e != cudaSuccess) return e;
  }
  // 2. main
  if (stages & 2) {
    cudaError_t e;
    if (a.k.bs_iter != nullptr) {
      // block-sparse exists for fp16 and head_dim <= 64 (checked by the C ABI)
      if (l.is_causal)
        e = l.is_dropout ? launch_main<64, false, true, true, true>(l, stream)
                         : launch_main<64, false, true, false, true>(l, stream);
      else
        e = l.is_dropout ? launch_main<64, false, false, true, true>(l, stream)
                         : launch_main<64, false, false, false, true>(l, stream);
    } else {
      e = l.dpad == 64 ? launch_d<64>(l, stream) : launch_d<128>(l, stream);
    }
    if (e != cudaSuccess) return e;
  }
  // 3. postprocess
  if ((stages & 4) && !a.one_launch) {
    const int64_t total = static_cast<int64_t>(a.total_q) * a.k.heads * (d / 8);
    if (total > 0) {
      const int threads = 256;
      const int blocks = static_cast<int>((total + threads - 1) / threads);
      cudaError_t e = launch(overlap_launches(l), l.is_bf16 ? bwd_postprocess_kernel<true> : bwd_postprocess_kernel<false>,
                             dim3(blocks), threads, 0, stream, a, l.dpad);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

}  // namespace fa
