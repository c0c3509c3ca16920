// Host-side launch interface between the C ABI (fa_api.cu) and the kernel translation units.
#pragma once
#include <atomic>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>
#include "fa_dropout.cuh"

namespace fa {

// Division of block indices (below 2^31) by a number known at launch, as a multiplication: with l = ceil(log2(div)) and mul =
// ceil(2^(31 + l) / div), which has 32 bits at most, n / div is the product's high part for every n < 2^31 (the error
// mul * div - 2^(31 + l) is below 2^l).
struct FastDiv {
  uint32_t mul, shift, div;
};
inline FastDiv fast_div(uint32_t div) {
  uint32_t l = 0;
  while ((uint64_t(1) << l) < div) ++l;
  return FastDiv{static_cast<uint32_t>(((uint64_t(1) << (31 + l)) + div - 1) / div), 31 + l, div};
}
#ifdef __CUDACC__
__host__ __device__ __forceinline__ uint32_t quotient(uint32_t n, const FastDiv& d) {
  return static_cast<uint32_t>((static_cast<uint64_t>(n) * d.mul) >> d.shift);
}
#endif

// Arguments shared by the forward and backward kernels (device pointers, sizes in elements).
struct KernelArgs {
  const int32_t* cu_seqlens_q;
  const int32_t* cu_seqlens_k;
  // Block-sparse: per (batch, key block of 256, 16-row block) iteration index of the reference
  // kernel, or -1 when the block is not in the layout; nullptr for dense attention.
  const int32_t* bs_iter;
  int32_t bs_rows16;   // row length of bs_iter: 16-row blocks per key block
  int32_t bs_kblocks;  // key blocks (of 256) per batch entry in bs_iter
  void* o;
  float* lse;
  int64_t o_row_stride, o_head_stride;
  int64_t lse_stride;
  int32_t batch, heads, head_dim;
  float scale;        // softmax_scale
  float scale_log2;   // softmax_scale * log2(e)
  float rp_keep;      // 1 / p_keep
  DropoutParams drop;
  int32_t* status;
  int32_t launch_id;  // non-zero serial number of this call: what an aborting CTA leaves in status[0]
  int32_t grid_tiles, grid_heads, grid_first;  // the backward's causal grids (see set_causal_grid)
  FastDiv tail_tiles, tail_pairs, tail_heads;  // the forward's (see set_tail_grid)
  int32_t tail_first;
  // Padded batches (fa_fwd_padded): every sequence has pad_rows rows, and the tokens of sequence b, one run of them, lie in rows
  // [cu_seqlens[2 b], cu_seqlens[2 b + 1]); a negative start: the launch has nothing to do.  0: packed tokens.
  int32_t pad_rows;
};

// Whether the blocks of a grid of (tiles, heads, batch) can be counted along its x dimension.  Beyond 2^31 - 1 blocks a
// launch has to keep its three dimensions (65535 sequences of 8 heads announced with 524289 keys, say), and so it does
// where heads or batch exceed theirs, which the launch refuses.
inline bool linear_grid(int64_t tiles, int64_t heads, int64_t batch) {
  return heads <= 65535 && batch <= 65535 && tiles * heads * batch <= 0x7fffffff;
}

// Block order of the causal grids, whose tiles differ in work by their number of keys (forward) or queries
// (backward): the last blocks to start should be short ones.  With the tiles of one (batch, head) pair after the other, the
// last pair's heavy tiles ran on while most SMs were done.
//
// Backward: the pairs come in sections of equal size whose streamed operands fit the L2 together (the first section takes
// what the division leaves over); within a section the heaviest tiles of all its pairs come first.  That also keeps
// the key tiles of a pair apart, which in the deterministic mode wait for one another (4 x 12 x 4096, deterministic, us, pair by
// pair -> sections: 884 -> 746 at d = 64, 1468 -> 1161 at d = 128).  Kernel clk: 2 x 4 x 16384 (d = 64) 1 356 000 ->
// 1 323 000; 4 x 32 x 3000 (d = 128) 1 857 000 -> 1 820 000; 16 x 12 x 1000 471 000 -> 450 000.
constexpr int64_t kSectionBytes = 32 << 20;
inline void set_causal_grid(KernelArgs* a, int tiles, int64_t bytes_per_pair) {
  const int64_t pairs = static_cast<int64_t>(a->heads) * a->batch;
  const int64_t most = kSectionBytes > bytes_per_pair ? kSectionBytes / bytes_per_pair : 1;
  const int64_t sections = (pairs + most - 1) / most;
  a->grid_tiles = tiles;
  a->grid_heads = static_cast<int32_t>((pairs + sections - 1) / sections);
  a->grid_first = static_cast<int32_t>(pairs - (sections - 1) * a->grid_heads);
}
#ifdef __CUDACC__
// Place of a block of such a linear grid; rank: 0 for the heaviest tile of a pair
__host__ __device__ __forceinline__ void causal_block(const KernelArgs& a, uint32_t block, int& rank, int& h, int& b) {
  const uint32_t tiles = a.grid_tiles, heads = a.heads;
  uint32_t n = a.grid_first, pair = 0, rest = block;
  if (rest >= n * tiles) {
    pair = n;
    rest -= n * tiles;
    n = a.grid_heads;
    const uint32_t section = rest / (n * tiles);
    pair += section * n;
    rest -= section * n * tiles;
  }
  rank = rest / n;
  pair += rest - rank * n;
  b = pair / heads;
  h = pair - b * heads;
}
#endif

// Forward: pair by pair, and only the last pairs heaviest tiles first, about three rounds of blocks (with fewer, the heaviest
// tile takes longer than the rest of the section).  Where all pairs come in sections, CTAs of one length share an SM and fall
// into step, and batches with short sequences run through their empty blocks with nothing beside them.  us, pair by pair -> sections
// -> here: 2 x 4 x 16384 (d = 64) 390 -> 318 -> 318, 4 x 12 x 4096 170 -> 152 -> 151, 32 x 12 x 1024 ragged 103.5 -> 104 -> 100,
// d = 128: 16 x 12 x 1000 94.8 -> 95.4 -> 93.3, 4 x 32 x 3000 321 -> 321 -> 312, 4 x 12 x 8192 711 -> 686 -> 683.  Uneven batches of
// 12 heads, d = 64 and 128: 31 x 256 and 1 x 8192 265 -> 305 -> 248 and 315 -> 292 -> 282 (with dropout 465 -> 415 -> 413), the
// long one first 224 -> 305 -> 236 and 261 -> 290 -> 268, 1 x 4096 and 63 x 128 171 -> 213 -> 179 and 159 -> 185 -> 163: what is
// lost there are the instructions that find a block's place, which an empty block waits for (with divisions 205 and 178).
constexpr int64_t kTailBlocks = 1024, kTailBytes = 64 << 20;
inline void set_tail_grid(KernelArgs* a, int tiles, int64_t bytes_per_pair) {
  const int64_t pairs = static_cast<int64_t>(a->heads) * a->batch;
  int64_t last = 1;  // (bytes_per_pair = 0: all pair by pair, which with one last pair comes to the same)
  if (bytes_per_pair > 0) last = kTailBlocks / tiles < kTailBytes / bytes_per_pair ? kTailBlocks / tiles : kTailBytes / bytes_per_pair;
  if (last > pairs) last = pairs;
  if (last < 1) last = 1;
  a->tail_tiles = fast_div(tiles);
  a->tail_pairs = fast_div(static_cast<uint32_t>(last));
  a->tail_heads = fast_div(a->heads);
  a->tail_first = static_cast<int32_t>((pairs - last) * tiles);
}
#ifdef __CUDACC__
__host__ __device__ __forceinline__ void tail_block(const KernelArgs& a, uint32_t block, int& rank, int& h, int& b) {
  const uint32_t first = a.tail_first;
  const bool last = block >= first;
  const uint32_t i = last ? block - first : block;
  const FastDiv n = last ? a.tail_pairs : a.tail_tiles;
  const uint32_t quot = quotient(i, n), rem = i - quot * n.div;
  const uint32_t pair = last ? static_cast<uint32_t>(a.heads) * a.batch - n.div + rem : quot;
  rank = last ? quot : rem;
  b = quotient(pair, a.tail_heads);
  h = pair - b * a.heads;
}
#endif

struct BwdArgs {
  KernelArgs k;
  const void* q; const void* kk; const void* v;       // raw pointers for the plain-load paths
  const void* o_in; const void* dout;
  int64_t q_row_stride, q_head_stride;
  int64_t do_row_stride, do_head_stride;
  void* dq; void* dk; void* dv;
  int64_t dq_row_stride, dq_head_stride, dk_row_stride, dk_head_stride, dv_row_stride, dv_head_stride;
  float* softmax_d;
  float* dq_accum;    // fp32 [total_q, heads, Dpad]
  // Deterministic mode: one ticket per (batch, head, 128-row query tile) = number of key tiles
  // that have added their dQ tile so far; nullptr = add in arrival order.
  int32_t* dq_tickets;
  // One query and one key tile per sequence: a block's dQ is the whole of it, which goes straight to dq, and softmax_d is its own
  // affair too; no accumulator, no other launch (see one_launch).
  bool one_launch;
  bool take_over;  // the grid has more blocks than SMs: a CTA goes on with blocks that have not started
  int32_t ticket_stride;  // tickets per (batch, head): ceil(max_seqlen_q / 128)
  int32_t total_q, total_k, max_seqlen_q, max_seqlen_k;
  float p_keep;
};

// Plain pointers of the decoding kernel (the tile kernels read through tensor maps).
constexpr int kDecodeMaxRows = 4;  // query rows per sequence it serves
struct DecodeArgs {
  const void* q; const void* k; const void* v;
  int64_t q_row_stride, q_head_stride, k_row_stride, k_head_stride, v_row_stride, v_head_stride;
  int32_t total_q, total_k;
};

struct FwdLaunch {
  CUtensorMap tm_q, tm_k, tm_v;
  CUtensorMap tm_o;  // output, boxes of 32 rows and out_box_columns columns, if any
  KernelArgs args;
  DecodeArgs decode;
  int32_t max_seqlen_q, max_seqlen_k, total_q;
  bool is_bf16, is_causal, is_dropout;
  int32_t dpad;  // 64 or 128
};

struct BwdLaunch {
  CUtensorMap tm_q, tm_k, tm_v, tm_do;
  CUtensorMap tm_dq;  // fp32 dQ accumulator [total_q, heads, dpad], 32-column boxes
  CUtensorMap tm_dk, tm_dv;  // outputs, boxes of 32 rows and grad_box_columns columns, if any
  BwdArgs args;
  bool is_bf16, is_causal, is_dropout;
  int32_t dpad;  // 64 or 128
  int32_t stage_mask;  // 0 = all; 1 preprocess, 2 main, 4 postprocess
  bool deterministic;
};

cudaError_t launch_fwd(const FwdLaunch& l, cudaStream_t stream);
int out_box_columns(const FwdLaunch& l);  // of the output that a warp of the tile kernel stores by TMA at once; 0: none
cudaError_t launch_fwd_padded(const FwdLaunch& l, cudaStream_t stream);
bool decode_serves(const FwdLaunch& l);  // whether launch_decode takes the call (l.decode apart)
cudaError_t launch_decode(const FwdLaunch& l, cudaStream_t stream);
// Columns of dK and dV that a warp of the backward's epilogue stores by TMA at once; 0: they leave by the LSU, without tensor maps.
// That is so at d = 64 without dropout and causal mask: there half as many bytes are stored as at d = 128, and
// the first P~ of the next block would wait for them behind dQ adds and loads (16 x 12 x 1024: 198 us by the LSU, 210 by TMA).
// Whole backward, us, by the LSU -> by TMA: 16 x 12 x 1000 causal (d = 128) 263 -> 255, 32 x 12 x 512 196 -> 189, 4 x 12 x 8192
// 2319 -> 2289; 8 x 12 x 512 with dropout (d = 64) 52.2 -> 50.2, 2 x 4 x 16384 causal 744 -> 733.
constexpr int grad_box_columns(int dpad, bool is_causal, bool is_dropout) {
  return dpad == 128 ? 64 : is_dropout ? 32 : is_causal ? 64 : 0;
}
// Whether the backward of a call is the main kernel alone, which then needs no workspace: one query tile, one key tile and no more
// blocks than SMs.  Such calls wait for the host and for launches.  Backward on the device, us, three kernels -> one: 12 x 128
// (d = 64) 19.5 -> 13.3, 12 x 12 x 128 causal (d = 128) 25.6 -> 19.4, 8 x 12 x 128 with dropout 23.5 -> 19.4; a training pass
// of the last 66.5 -> 60.2.  softmax_d and dq, made beside each tile, are what the tile then waits for: with several query tiles
// (12 x 2048 queries, 100 keys 44 -> 95) or more blocks than SMs (32 x 12 x 128 with dropout 34 -> 44) three kernels are
// faster.  So are they on the device at d = 128 with few rows (8 x 40: 21.5 -> 22.6-24.4, inputs in DRAM), but the pass waits for the host
// (64.6 -> 56.2).  Block-sparse calls and single stages keep the three.
constexpr int kOneLaunchBlocks = 148;
inline bool one_launch(int max_seqlen_q, int max_seqlen_k, int64_t pairs, bool sparse, int stage_mask) {
  return max_seqlen_q <= 128 && max_seqlen_k <= 128 && pairs <= kOneLaunchBlocks && !sparse && stage_mask == 0;
}
cudaError_t launch_bwd(const BwdLaunch& l, cudaStream_t stream);
cudaError_t launch_sdmask(void* s_out, int64_t s_rows, int64_t s_cols, const void* q, const void* k,
                          int64_t q_row_stride, int64_t q_head_stride, int64_t k_row_stride,
                          int64_t k_head_stride, const KernelArgs& a, int max_seqlen_q, int max_seqlen_k,
                          bool bf16, bool causal, bool dropout, cudaStream_t stream);
cudaError_t launch_philox_probe(uint32_t* out, int n, unsigned long long seed, unsigned long long offset,
                                int rounds, int mode, cudaStream_t stream);
cudaError_t launch_bs_table(int32_t* table, const int32_t* blockmask, const int32_t* cu_q,
                            const int32_t* cu_k, int batch, int nk, int nr, void* o, int64_t o_row_bytes,
                            int total_q, int max_seqlen_q, cudaStream_t stream);
cudaError_t launch_convert_blockmask(int32_t* out, const void* layout, int elem_bytes, bool is_float, int64_t row_stride,
                                     int64_t col_stride, int nrow, int ncol, bool causal, cudaStream_t stream);
cudaError_t launch_dropout_mask(uint8_t* out, int b, int h, const DropoutParams& dp, bool causal,
                                int sq, int sk, const int32_t* bs_iter, int bs_kblocks,
                                int bs_rows16, cudaStream_t stream);

cudaError_t launch_gather_rows(const void* src, const int64_t* indices, void* dst, int64_t n_rows,
                               int64_t src_rows, int64_t row_bytes, cudaStream_t stream);
cudaError_t launch_scatter_rows(const void* src, const int64_t* indices, void* dst, int64_t n_src_rows,
                                int64_t n_dst_rows, int64_t row_bytes, int32_t* inverse,
                                cudaStream_t stream);

cudaError_t launch_mask_index(const uint8_t* mask, int batch, int seqlen, int32_t* counts, int32_t* cu_seqlens,
                              int64_t* indices, int32_t* summary, cudaStream_t stream);
cudaError_t launch_mask_bounds(const uint8_t* mask, int batch, int seqlen, int32_t* bounds, int32_t* summary,
                               cudaStream_t stream);

cudaError_t launch_rotary_qkv(const void* qkv, void* out, const float* cos_t, const float* sin_t,
                              int64_t rows, int seqlen, int heads, int d, bool bf16, bool conj,
                              cudaStream_t stream);

// Raises the dynamic shared-memory limit of `kernel` the first time it is launched on a device
// (the attribute belongs to the device's context; setting it on every launch costs microseconds).
// `done` is the caller's per-kernel flag array, one entry per device: kernels that differ only in
// template arguments have the same function type, so the flags cannot live in this template.
constexpr int kMaxDevices = 64;
using SmemLimitFlags = std::atomic<unsigned char>[kMaxDevices];
template <typename Kernel>
inline cudaError_t set_smem_limit_once(Kernel kernel, int bytes, SmemLimitFlags& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < kMaxDevices && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && dev >= 0 && dev < kMaxDevices) done[dev].store(1, std::memory_order_release);
  return e;
}

}  // namespace fa
