// Forward for a handful of query rows per sequence (a decoding step against cached keys and values).
//
// Bound by the HBM with one row: every key and value is read once and used for at most kDecodeMaxRows rows, 2
// to 8 FLOP a byte.  The tile kernel (fa_fwd_sm100.cu) works on 128 query rows: with one row it multiplies
// and exponentiates 127 rows of padding and has batch x heads CTAs whatever the length of the
// sequences.  Here
//   * the keys of a (batch, head) are split over the CTAs of a cluster (grid.x = cluster size = 1, 2,
//     4 or 8), whose partial results meet in distributed shared memory: one launch, no workspace;
//   * a warp reads whole rows of K and V with 16-byte loads (D / 8 lanes per row), kLoads rows of each
//     per lane group in flight, and 16 warps per SM cover the latency;
//   * every lane group keeps its own running maximum, sum and fp32 accumulator; they are merged over
//     the warp by shuffles, over the CTA in shared memory and over the cluster at the end.
// Scores, probabilities, sums and outputs stay in fp32 (the tile kernel rounds P to 16 bits before P*V).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "fa_kernels.h"
#include "fa_math.cuh"
#include "sm100_prims.cuh"

namespace fa {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

template <bool BF16>
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 x;
    if constexpr (BF16) x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    else x = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    f[2 * i] = x.x;
    f[2 * i + 1] = x.y;
  }
}

__device__ __forceinline__ uint4 load16_stream(const uint16_t* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// fp32 word at the same shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ float cluster_load(uint32_t saddr, uint32_t rank) {
  uint32_t remote;
  float v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(saddr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}

// Weight of a partial result with maximum m_i once the maximum is m (raw score units).
__device__ __forceinline__ float merge_weight(float m_i, float m, float scale_log2) {
  return m_i == -INFINITY ? 0.f : ex2f((m_i - m) * scale_log2);
}

// D: head_dim; R: query rows a CTA serves (rows past the sequence's length are computed on zeros)
template <int D, bool BF16, int R>
__global__ void __launch_bounds__(kThreads, 2) fa_decode_kernel(const KernelArgs a, const DecodeArgs t) {
  constexpr int kLanes = D / 8;           // lanes per row of K or V
  constexpr int kGroups = 32 / kLanes;    // rows a warp reads with one load
  constexpr int kLoads = R == 1 ? 8 : 4;  // rows of K and of V in flight per lane group
  constexpr int kStep = kGroups * kLoads; // keys per warp and iteration
  __shared__ float sm_acc[kWarps][R][D];
  __shared__ float sm_m[kWarps][R], sm_l[kWarps][R];
  __shared__ float part_acc[R][D], part_m[R], part_l[R];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = lane / kLanes, c = (lane % kLanes) * 8;
  const int h = blockIdx.y, b = blockIdx.z;
  const int split = blockIdx.x, n_splits = gridDim.x;
  const int q_start = a.cu_seqlens_q[b];
  const int sq = min(a.cu_seqlens_q[b + 1] - q_start, R);
  const int k_start = a.cu_seqlens_k[b];
  const int sk = a.cu_seqlens_k[b + 1] - k_start;
  if (sq <= 0) return;  // the same in every CTA of the cluster

  // this CTA's keys, in whole steps of its eight warps
  constexpr int kUnit = kStep * kWarps;
  const int per = (max(sk, 0) + n_splits * kUnit - 1) / (n_splits * kUnit) * kUnit;
  const int k_begin = min(split * per, max(sk, 0)), k_end = min(k_begin + per, max(sk, 0));

  float q[R][8], acc[R][8], m_run[R], l_run[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    uint4 v = make_uint4(0, 0, 0, 0);
    // rows outside the tensor read as zero, as they do through a tensor map
    if (r < sq && static_cast<uint32_t>(q_start + r) < static_cast<uint32_t>(t.total_q))
      v = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(t.q) +
                                          static_cast<int64_t>(q_start + r) * t.q_row_stride + h * t.q_head_stride + c);
    unpack8<BF16>(v, q[r]);
    m_run[r] = -INFINITY;
    l_run[r] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[r][i] = 0.f;
  }
  const uint16_t* kp = reinterpret_cast<const uint16_t*>(t.k) + h * t.k_head_stride + c;
  const uint16_t* vp = reinterpret_cast<const uint16_t*>(t.v) + h * t.v_head_stride + c;

  for (int key0 = k_begin + warp * kStep; key0 < k_end; key0 += kUnit) {
    uint4 kv[kLoads], vv[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int key = key0 + u * kGroups + grp;
      const uint32_t row = static_cast<uint32_t>(k_start + key);
      kv[u] = make_uint4(0, 0, 0, 0);
      if (key < k_end && row < static_cast<uint32_t>(t.total_k)) kv[u] = load16_stream(kp + row * t.k_row_stride);
    }
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int key = key0 + u * kGroups + grp;
      const uint32_t row = static_cast<uint32_t>(k_start + key);
      vv[u] = make_uint4(0, 0, 0, 0);
      if (key < k_end && row < static_cast<uint32_t>(t.total_k)) vv[u] = load16_stream(vp + row * t.v_row_stride);
    }
    float s[R][kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      float f[8];
      unpack8<BF16>(kv[u], f);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float x = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) x = fmaf(q[r][i], f[i], x);
        s[r][u] = x;
      }
    }
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int u = 0; u < kLoads; ++u) s[r][u] += __shfl_xor_sync(0xffffffffu, s[r][u], off);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float m_new = m_run[r];
#pragma unroll
      for (int u = 0; u < kLoads; ++u) {
        if (key0 + u * kGroups + grp >= k_end) s[r][u] = -INFINITY;
        m_new = fmaxf(m_new, s[r][u]);
      }
      const float alpha = merge_weight(m_run[r], m_new, a.scale_log2);
      m_run[r] = m_new;
      const float mc = m_new == -INFINITY ? 0.f : m_new * a.scale_log2;
      l_run[r] *= alpha;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[r][i] *= alpha;
#pragma unroll
      for (int u = 0; u < kLoads; ++u) {
        s[r][u] = ex2f(fmaf(s[r][u], a.scale_log2, -mc));
        l_run[r] += s[r][u];
      }
    }
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      float f[8];
      unpack8<BF16>(vv[u], f);
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[r][i] = fmaf(s[r][u], f[i], acc[r][i]);
    }
  }

  // lane groups of the warp
#pragma unroll
  for (int off = kLanes; off < 32; off <<= 1)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float m_other = __shfl_xor_sync(0xffffffffu, m_run[r], off);
      const float m = fmaxf(m_run[r], m_other);
      const float w = merge_weight(m_run[r], m, a.scale_log2);
      l_run[r] *= w;
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], off);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        acc[r][i] *= w;
        acc[r][i] += __shfl_xor_sync(0xffffffffu, acc[r][i], off);
      }
      m_run[r] = m;
    }
  if (lane < kLanes) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int i = 0; i < 8; ++i) sm_acc[warp][r][c + i] = acc[r][i];
      if (lane == 0) { sm_m[warp][r] = m_run[r]; sm_l[warp][r] = l_run[r]; }
    }
  }
  __syncthreads();

  // warps of the CTA, then the CTAs of the cluster: element (r, col) by one thread
  for (int e = tid; e < R * D; e += kThreads) {
    const int r = e / D, col = e % D;
    float m = -INFINITY, l = 0.f, x = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) m = fmaxf(m, sm_m[w][r]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = merge_weight(sm_m[w][r], m, a.scale_log2);
      l = fmaf(f, sm_l[w][r], l);
      x = fmaf(f, sm_acc[w][r][col], x);
    }
    part_acc[r][col] = x;
    if (col == 0) { part_m[r] = m; part_l[r] = l; }
  }
  if (n_splits > 1) cluster_barrier(); else __syncthreads();
  if (split == 0) {
    for (int e = tid; e < R * D; e += kThreads) {
      const int r = e / D, col = e % D;
      if (r >= sq) continue;
      float m = part_m[r], l = part_l[r], x = part_acc[r][col];
      if (n_splits > 1) {
        for (int s = 1; s < n_splits; ++s) m = fmaxf(m, cluster_load(smem_u32(&part_m[r]), s));
        const float f0 = merge_weight(part_m[r], m, a.scale_log2);
        l *= f0;
        x *= f0;
        for (int s = 1; s < n_splits; ++s) {
          const float f = merge_weight(cluster_load(smem_u32(&part_m[r]), s), m, a.scale_log2);
          l = fmaf(f, cluster_load(smem_u32(&part_l[r]), s), l);
          x = fmaf(f, cluster_load(smem_u32(&part_acc[r][col]), s), x);
        }
      }
      const bool bad_sum = (l == 0.f) || (l != l);
      const float o = x * (bad_sum ? 1.f : (1.f / l) * a.rp_keep);
      uint16_t* dst = reinterpret_cast<uint16_t*>(a.o) + static_cast<int64_t>(q_start + r) * a.o_row_stride +
                      static_cast<int64_t>(h) * a.o_head_stride + col;
      *dst = static_cast<uint16_t>(pack_lowp<BF16>(o, o) & 0xffffu);
      if (col == 0)
        a.lse[(static_cast<int64_t>(b) * a.heads + h) * a.lse_stride + r] = bad_sum ? -INFINITY : m * a.scale + __logf(l);
    }
  }
  if (n_splits > 1) cluster_barrier();  // the other CTAs' shared memory stays until it has been read
}

template <int D, bool BF16, int R>
cudaError_t launch_one(const FwdLaunch& l, int splits, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(splits, l.args.heads, l.args.batch);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = splits;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fa_decode_kernel<D, BF16, R>, l.args, l.decode);
}

template <int D>
cudaError_t launch_d(const FwdLaunch& l, int splits, cudaStream_t stream) {
  if (l.max_seqlen_q == 1)
    return l.is_bf16 ? launch_one<D, true, 1>(l, splits, stream) : launch_one<D, false, 1>(l, splits, stream);
  return l.is_bf16 ? launch_one<D, true, kDecodeMaxRows>(l, splits, stream)
                   : launch_one<D, false, kDecodeMaxRows>(l, splits, stream);
}

}  // namespace

// Where this kernel is the faster one (the tile kernel takes the other calls).  It reads K and V at the rate of the
// memory with any grid.  The tile kernel comes near that rate when the (batch, head) pairs fill a round of it,
// 112 to 148 pairs with one CTA per SM or 223 to 296 with two, and the sequences are long enough for its prologue and
// short enough for the memory's rate not to have been reached here (1024 keys to 64 * head_dim, or twice that with
// more rows; 2048 at d = 16).  Four rows take up to four times the arithmetic of one per byte, which bounds the
// kernel at d = 64 and 128 once the grid fills the chip.  us here / in the tile kernel, every sequence of
// `keys` keys, bf16:
//                pairs  keys  64        256       1024       4096       8192
//   1 row   d = 32    144   3.8/6.3   4.1/7.2    15/13      31/38      47/71
//           d = 64     64   3.9/6.0   4.3/6.7   6.9/13      17/37      32/71
//                     144   4.0/6.4   4.4/7.4    16/14      46/40      71/72
//                     192   4.2/7.4   5.2/8.8    19/18      44/58     75/107
//                     288   4.4/7.7   5.7/9.2    29/19      67/59    114/109
//                    1024    11/19     17/23     49/59    165/195    325/385
//           d = 128   144   3.9/7.2   5.9/8.2    23/17      70/54    117/100
//                     192   4.3/8.2   7.7/10     27/25      74/85    134/157
//                    1024    16/26     32/39     84/97    311/351    620/693
//   4 rows  d = 32    144   4.4/6.4   5.0/7.1    18/13      43/38      64/71
//                    1024    14/19     18/22     41/55    127/181    240/350
//           d = 64     64   4.2/5.8   5.9/6.5    10/13      28/37      47/70
//                     144   4.8/6.9   6.2/7.4    23/14      66/40     105/72
//                    1024    15/19     26/23     72/59    250/204    501/401
//           d = 128    64   4.9/6.6   8.8/7.4    16/16      53/52      90/97
//                     144   5.0/6.8   9.6/7.7    40/17     122/54    210/100
//                    1024    23/26     53/38    149/98    543/359   1078/710
static bool decode_is_faster(int head_dim, int rows, int64_t pairs, int keys) {
  constexpr int kSms = 148;
  if (rows == 1 || head_dim <= 32) {
    const bool full_round = (pairs > kSms * 3 / 4 && pairs <= kSms) || (pairs > kSms * 3 / 2 && pairs <= 2 * kSms);
    const int longest = max(2048, (rows == 1 ? 64 : 128) * head_dim);
    return !(full_round && keys >= 1024 && keys <= longest);
  }
  if (pairs <= kSms / 2) return head_dim == 64 || keys <= 64 || keys >= 512;
  return keys <= (head_dim == 64 ? 256 : 64);
}

bool decode_serves(const FwdLaunch& l) {
  return l.max_seqlen_q <= kDecodeMaxRows && !l.is_dropout && !l.is_causal && l.args.bs_iter == nullptr &&
         decode_is_faster(l.args.head_dim, l.max_seqlen_q, static_cast<int64_t>(l.args.batch) * l.args.heads, l.max_seqlen_k);
}

// Key ranges per (batch, head): doubled while there are fewer CTAs than four per SM (two are resident;
// ragged sequences want a second round to even out) and a CTA keeps at least 256 keys.
static int decode_splits(int batch, int heads, int max_seqlen_k) {
  const int64_t pairs = static_cast<int64_t>(batch) * heads;
  int splits = 1;
  while (splits < 8 && pairs * splits < 4 * 148 && max_seqlen_k / (2 * splits) >= 256) splits *= 2;
  return splits;
}

cudaError_t launch_decode(const FwdLaunch& l, cudaStream_t stream) {
  const int splits = decode_splits(l.args.batch, l.args.heads, l.max_seqlen_k);
  switch (l.args.head_dim) {
    case 16: return launch_d<16>(l, splits, stream);
    case 32: return launch_d<32>(l, splits, stream);
    case 64: return launch_d<64>(l, splits, stream);
    default: return launch_d<128>(l, splits, stream);
  }
}

}  // namespace fa
