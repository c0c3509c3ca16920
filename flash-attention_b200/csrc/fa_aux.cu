// Small helper kernels: dropout-mask dump (test hook), block-sparse iteration table.
#include <algorithm>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <curand_kernel.h>
#include "fa_kernels.h"

namespace fa {

namespace {

// One thread per (row, 16-column group).
__global__ void dropout_mask_kernel(uint8_t* out, int b, int h, DropoutParams dp, bool causal,
                                    int sq, int sk, const int32_t* bs_iter, int bs_kblocks,
                                    int bs_rows16) {
  const int groups = (sk + 15) / 16;
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<int64_t>(sq) * groups) return;
  const int i = static_cast<int>(idx / groups);
  const int jg0 = static_cast<int>(idx % groups) * 16;
  const int64_t bh_sub = (static_cast<int64_t>(b) * dp.heads_total + dp.head_offset + h) * 256;
  int64_t it;
  if (bs_iter) {
    it = bs_iter[(static_cast<int64_t>(b) * bs_kblocks + (jg0 >> 8)) * bs_rows16 + (i >> 4)];
  } else {
    it = fa_iter_index(causal, jg0 >> dp.n_shift, i >> 4, (sq + 15) >> 4, dp.n_shift);
  }
  const uint32_t keep = fa_dropout_keep16(dp, bh_sub, i, jg0, it);
  for (int o = 0; o < 16 && jg0 + o < sk; ++o)
    out[static_cast<int64_t>(i) * sk + jg0 + o] = (keep >> o) & 1u;
}

// Block-sparse iteration table.  The converted block mask lists, for each 256-column key block,
// the 16-row query blocks to visit in ascending order (value = 4 * row_block + flags, -1 ends the
// list).  The reference walks key blocks in order and, inside one, the list until it ends or
// reaches a row block at or beyond the sequence's query length
// (csrc/flash_attn/src/fmha_block_fprop_kernel_1xN.h:90-100, :209, :486); key blocks at or beyond
// the key length are not visited at all (:88).  table[b][kb][rb] = number of blocks visited
// before (kb, rb), or -1 when (kb, rb) is not visited.
//
// One CTA per (key block, batch entry).  It is a few KB of integers, bound by latency: a warp finds the
// end of a list with coalesced 32-entry reads and a ballot, the CTA's eight warps share the lists in
// front of its own, and nothing is serial but that sum.  (One CTA per batch entry with a thread per list
// walked 256 dependent loads: 28 us at 4 x 4096 tokens, 6 us now.)
constexpr int kTableThreads = 256;

// Length of the visited prefix of one list (all lanes return it).
__device__ __forceinline__ int visited_prefix(const int32_t* row, int nr, int sq, int lane) {
  for (int c = 0; c < nr; c += 32) {
    const int32_t v = c + lane < nr ? row[c + lane] : -1;
    const unsigned stop = __ballot_sync(0xffffffffu, v < 0 || (v >> 2) * 16 >= sq);
    if (stop != 0u) return c + __ffs(stop) - 1;
  }
  return nr;
}

// Output rows no attention CTA writes (rows outside every sequence, and rows at or beyond the 128-row
// tiles that max_seqlen_q covers) are zero in a block-sparse call (fmha_api.cpp:519 starts from
// o = 0); zeroing the few there are replaces a pass over the whole tensor.  A token buffer of fixed size
// may leave most of its rows unused: CTAs of their own share the rows in front of and behind the sequences, one
// per 32 KB of o up to four per SM (those that find nothing to do read two integers).  12 x 64 heads,
// 4 x 512 tokens, 100 000 unused rows, us of the whole call: 64 with the full pass, 2462 with one CTA, 42 so.
struct ZeroRows {
  uint4* o;          // nullptr: nothing to zero
  int64_t row_vecs;  // 16-byte units per (contiguous) row
  int32_t total_q, max_q_tiles;  // rows per sequence that the attention grid covers
};
constexpr int kZeroCtaBytes = 32768, kZeroMaxCtas = 4 * 148;

__device__ __forceinline__ void zero_rows(const ZeroRows& z, int64_t first, int64_t last, int part, int parts) {
  for (int64_t i = first * z.row_vecs + static_cast<int64_t>(part) * blockDim.x + threadIdx.x; i < last * z.row_vecs;
       i += static_cast<int64_t>(parts) * blockDim.x)
    z.o[i] = make_uint4(0, 0, 0, 0);
}

// CTAs [0, nk * batch): key block bid % nk of batch entry bid / nk; the CTAs behind them zero rows.
__global__ void __launch_bounds__(kTableThreads)
bs_table_kernel(int32_t* table, const int32_t* blockmask, const int32_t* cu_q, const int32_t* cu_k, int nk, int nr,
                int batch, ZeroRows z) {
  __shared__ int sum[kTableThreads / 32];
  const int b = blockIdx.x / nk, kb = blockIdx.x - b * nk;
  if (b >= batch) {
    const int part = blockIdx.x - nk * batch, parts = gridDim.x - nk * batch;
    zero_rows(z, 0, min(cu_q[0], z.total_q), part, parts);
    zero_rows(z, max(cu_q[batch], 0), z.total_q, part, parts);
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sq = cu_q[b + 1] - cu_q[b];
  const int sk = cu_k[b + 1] - cu_k[b];
  if (z.o != nullptr)
    zero_rows(z, static_cast<int64_t>(cu_q[b]) + min(sq, z.max_q_tiles), min(cu_q[b + 1], z.total_q), kb, nk);
  int32_t* trow = table + (static_cast<int64_t>(b) * nk + kb) * nr;
  for (int i = threadIdx.x; i < nr; i += kTableThreads) trow[i] = -1;
  if (kb * 256 >= sk) return;
  int before = 0;
  for (int k = warp; k < kb; k += kTableThreads / 32)
    before += visited_prefix(blockmask + static_cast<int64_t>(k) * nr, nr, sq, lane);
  if (lane == 0) sum[warp] = before;
  __syncthreads();  // also orders the -1 fill before the entries below
  before = 0;
#pragma unroll
  for (int w = 0; w < kTableThreads / 32; ++w) before += sum[w];
  const int32_t* row = blockmask + static_cast<int64_t>(kb) * nr;
  const int n = visited_prefix(row, nr, sq, lane);
  for (int c = threadIdx.x; c < n; c += kTableThreads) {
    const int rb = row[c] >> 2;
    if (rb < nr) trow[rb] = before + c;
  }
}

// 0/1 layout (nrow, ncol) -> per-column visit lists (flash_blocksparse_attn_interface.py:8-40 of the
// reference): out[c] lists 4 * r in ascending order for every set (r, c), plus 1 when c is the first set
// column of row r and plus 2 when it is the last, then -1.  causal drops the blocks that lie entirely
// above the diagonal first.  One CTA per column; rows are compacted 256 at a time with ballots.  Latency
// bound like the table above (it replaces two dozen framework launches, 400 us of host time).
template <typename T>
__device__ __forceinline__ bool layout_set(const T* m, int64_t row_stride, int64_t col_stride, int r, int c, T value_bits,
                                           bool causal) {
  return (m[r * row_stride + c * col_stride] & value_bits) != 0 && !(causal && 256 * c > 16 * r + 15);
}

template <typename T>
__global__ void __launch_bounds__(kTableThreads)
convert_blockmask_kernel(int32_t* out, const T* m, int64_t row_stride, int64_t col_stride, int nrow, int ncol,
                         T value_bits, bool causal) {
  __shared__ int warp_count[2][kTableThreads / 32];
  const int c = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int32_t* dst = out + static_cast<int64_t>(c) * nrow;
  int done = 0, buf = 0;
  for (int r0 = 0; r0 < nrow; r0 += kTableThreads, buf ^= 1) {
    const int r = r0 + threadIdx.x;
    const bool on = r < nrow && layout_set(m, row_stride, col_stride, r, c, value_bits, causal);
    const unsigned bits = __ballot_sync(0xffffffffu, on);
    if (lane == 0) warp_count[buf][warp] = __popc(bits);
    __syncthreads();  // double-buffered counts: one barrier per chunk
    int pos = done;
#pragma unroll
    for (int w = 0; w < kTableThreads / 32; ++w) {
      const int n = warp_count[buf][w];
      if (w < warp) pos += n;
      done += n;
    }
    if (on) {
      int first = 0, last = ncol - 1;
      while (!layout_set(m, row_stride, col_stride, r, first, value_bits, causal)) ++first;  // ends at c at the latest
      while (!layout_set(m, row_stride, col_stride, r, last, value_bits, causal)) --last;
      dst[pos + __popc(bits & ((1u << lane) - 1u))] = 4 * r + (first == c ? 1 : 0) + (last == c ? 2 : 0);
    }
  }
  for (int i = done + threadIdx.x; i < nrow; i += kTableThreads) dst[i] = -1;
}

// return_softmax output (test aid): s[b, h, i, j] = softmax probability of key j for query i,
// recomputed from q, k and the saved LSE on the CUDA cores, with the sign bit set where dropout
// dropped the entry.  The reference stores un-normalised values in its MMA fragment order
// (csrc/flash_attn/src/fmha/gmem_tile.h:289-405); this writes the documented (batch, heads,
// seqlen_q, seqlen_k) layout with normalised values.  One thread per (query, 16-key group).
template <bool BF16>
__global__ void sdmask_kernel(void* s_out, int64_t s_rows, int64_t s_cols, const void* q, const void* k,
                              int64_t q_row_stride, int64_t q_head_stride, int64_t k_row_stride,
                              int64_t k_head_stride, const KernelArgs a, bool causal, bool dropout) {
  const int b = blockIdx.z, h = blockIdx.y;
  const int q_start = a.cu_seqlens_q[b], sq = a.cu_seqlens_q[b + 1] - q_start;
  const int k_start = a.cu_seqlens_k[b], sk = a.cu_seqlens_k[b + 1] - k_start;
  const int groups = (sk + 15) / 16;
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<int64_t>(sq) * groups) return;
  const int i = static_cast<int>(idx / groups);
  const int jg0 = static_cast<int>(idx % groups) * 16;
  const int d = a.head_dim;
  const uint16_t* qrow = reinterpret_cast<const uint16_t*>(q) + (q_start + i) * q_row_stride + h * q_head_stride;
  const float lse = a.lse[(static_cast<int64_t>(b) * a.heads + h) * a.lse_stride + i];
  int64_t it = 0;
  bool in_layout = true;
  if (a.bs_iter) {
    it = (i >> 4) < a.bs_rows16
             ? a.bs_iter[(static_cast<int64_t>(b) * a.bs_kblocks + (jg0 >> 8)) * a.bs_rows16 + (i >> 4)] : -1;
    in_layout = it >= 0;
  } else {
    it = fa_iter_index(causal, jg0 >> a.drop.n_shift, i >> 4, (sq + 15) >> 4, a.drop.n_shift);
  }
  uint32_t keep = 0xffffu;
  if (dropout) {
    const int64_t bh_sub = (static_cast<int64_t>(b) * a.drop.heads_total + a.drop.head_offset + h) * 256;
    keep = fa_dropout_keep16(a.drop, bh_sub, i, jg0, it < 0 ? 0 : it);
  }
  uint16_t* out = reinterpret_cast<uint16_t*>(s_out) + ((static_cast<int64_t>(b) * a.heads + h) * s_rows + i) * s_cols;
  for (int o = 0; o < 16 && jg0 + o < sk; ++o) {
    const int j = jg0 + o;
    const uint16_t* krow = reinterpret_cast<const uint16_t*>(k) + (k_start + j) * k_row_stride + h * k_head_stride;
    float acc = 0.f;
    for (int c = 0; c < d; ++c) {
      float qv, kv;
      if constexpr (BF16) {
        qv = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(qrow)[c]);
        kv = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(krow)[c]);
      } else {
        qv = __half2float(reinterpret_cast<const __half*>(qrow)[c]);
        kv = __half2float(reinterpret_cast<const __half*>(krow)[c]);
      }
      acc += qv * kv;
    }
    const bool visible = in_layout && (!causal || j <= i);
    float p = visible ? __expf(acc * a.scale - lse) : 0.f;
    if (!((keep >> o) & 1u)) p = -p;
    if (j < s_cols) {
      if constexpr (BF16) reinterpret_cast<__nv_bfloat16*>(out)[j] = __float2bfloat16(p);
      else reinterpret_cast<__half*>(out)[j] = __float2half(p);
    }
  }
}

// Philox self-check: thread i writes the four output words for (seed, subsequence i, offset).
// mode 0: this library's round function run `rounds` times with the counter layout of the
// attention kernels; mode 1: cuRAND's Philox4_32_10 device generator (10 rounds) as an
// independent implementation of the same generator.
__global__ void philox_probe_kernel(uint32_t* out, int n, unsigned long long seed,
                                    unsigned long long offset, int rounds, int mode) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t c[4];
  if (mode == 1) {
    curandStatePhilox4_32_10_t st;
    curand_init(seed, static_cast<unsigned long long>(i), offset, &st);
    const uint4 r = curand4(&st);
    c[0] = r.x; c[1] = r.y; c[2] = r.z; c[3] = r.w;
  } else {
    const unsigned long long ctr = offset / 4;
    c[0] = static_cast<uint32_t>(ctr);
    c[1] = static_cast<uint32_t>(ctr >> 32);
    c[2] = static_cast<uint32_t>(i);
    c[3] = 0u;
    uint32_t k0 = static_cast<uint32_t>(seed), k1 = static_cast<uint32_t>(seed >> 32);
    for (int r = 0; r < rounds; ++r) {
      philox_round(c, k0, k1);
      k0 += 0x9E3779B9u;
      k1 += 0xBB67AE85u;
    }
  }
  for (int k = 0; k < 4; ++k) out[4 * i + k] = c[k];
}

}  // namespace

cudaError_t launch_sdmask(void* s_out, int64_t s_rows, int64_t s_cols, const void* q, const void* k,
                          int64_t q_row_stride, int64_t q_head_stride, int64_t k_row_stride,
                          int64_t k_head_stride, const KernelArgs& a, int max_seqlen_q, int max_seqlen_k,
                          bool bf16, bool causal, bool dropout, cudaStream_t stream) {
  const int64_t n = static_cast<int64_t>(max_seqlen_q) * ((max_seqlen_k + 15) / 16);
  if (n == 0) return cudaSuccess;
  dim3 grid(static_cast<unsigned>((n + 127) / 128), a.heads, a.batch);
  if (bf16)
    sdmask_kernel<true><<<grid, 128, 0, stream>>>(s_out, s_rows, s_cols, q, k, q_row_stride, q_head_stride,
                                                  k_row_stride, k_head_stride, a, causal, dropout);
  else
    sdmask_kernel<false><<<grid, 128, 0, stream>>>(s_out, s_rows, s_cols, q, k, q_row_stride, q_head_stride,
                                                   k_row_stride, k_head_stride, a, causal, dropout);
  return cudaGetLastError();
}

cudaError_t launch_philox_probe(uint32_t* out, int n, unsigned long long seed, unsigned long long offset,
                                int rounds, int mode, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  philox_probe_kernel<<<(n + 127) / 128, 128, 0, stream>>>(out, n, seed, offset, rounds, mode);
  return cudaGetLastError();
}

cudaError_t launch_bs_table(int32_t* table, const int32_t* blockmask, const int32_t* cu_q,
                            const int32_t* cu_k, int batch, int nk, int nr, void* o, int64_t o_row_bytes,
                            int total_q, int max_seqlen_q, cudaStream_t stream) {
  const ZeroRows z{static_cast<uint4*>(o), o_row_bytes / 16, total_q, (max_seqlen_q + 127) / 128 * 128};
  int64_t zero_ctas = 0;
  if (o != nullptr) zero_ctas = std::min<int64_t>(o_row_bytes * total_q / kZeroCtaBytes + 1, kZeroMaxCtas);
  bs_table_kernel<<<static_cast<unsigned>(nk * batch + zero_ctas), kTableThreads, 0, stream>>>(table, blockmask, cu_q, cu_k,
                                                                                               nk, nr, batch, z);
  return cudaGetLastError();
}

cudaError_t launch_convert_blockmask(int32_t* out, const void* layout, int elem_bytes, bool is_float, int64_t row_stride,
                                     int64_t col_stride, int nrow, int ncol, bool causal, cudaStream_t stream) {
  if (nrow <= 0 || ncol <= 0) return cudaSuccess;
  // an element is set when it differs from zero: any bit, without the sign of a floating-point zero
#define FA_CONVERT(T)                                                                                             \
  convert_blockmask_kernel<T><<<ncol, kTableThreads, 0, stream>>>(                                                 \
      out, static_cast<const T*>(layout), row_stride, col_stride, nrow, ncol,                                      \
      static_cast<T>(is_float ? static_cast<T>(~T(0)) >> 1 : static_cast<T>(~T(0))), causal)
  switch (elem_bytes) {
    case 1: FA_CONVERT(uint8_t); break;
    case 2: FA_CONVERT(uint16_t); break;
    case 4: FA_CONVERT(uint32_t); break;
    default: FA_CONVERT(uint64_t); break;
  }
#undef FA_CONVERT
  return cudaGetLastError();
}

cudaError_t launch_dropout_mask(uint8_t* out, int b, int h, const DropoutParams& dp, bool causal,
                                int sq, int sk, const int32_t* bs_iter, int bs_kblocks,
                                int bs_rows16, cudaStream_t stream) {
  const int64_t n = static_cast<int64_t>(sq) * ((sk + 15) / 16);
  if (n == 0) return cudaSuccess;
  const int threads = 256;
  const int blocks = static_cast<int>((n + threads - 1) / threads);
  dropout_mask_kernel<<<blocks, threads, 0, stream>>>(out, b, h, dp, causal, sq, sk, bs_iter,
                                                      bs_kblocks, bs_rows16);
  return cudaGetLastError();
}

}  // namespace fa
