// Which kernel serves a call: rules on sizes alone, for the launches (and for tests on the host, which compile this file).
#pragma once
#include <algorithm>
#include <climits>
#include "fa_kernels.h"

namespace fa {

constexpr int kBlockM = 128;  // query rows of a tile
constexpr int kBlockN = 128;  // key rows of a tile

// How a grid is laid out and worked on.  kPlain: (tiles, heads, batch).  kLinear: one-dimensional, causal ones with the order of
// set_tail_grid.  kTake: kLinear, and a CTA goes on with blocks that have not started (see take_over_pays).
enum Order { kPlain, kLinear, kTake };

// Announced lengths above `times` the actual ones on average: the grid consists mostly of blocks without queries.
inline bool uneven(const FwdLaunch& l, int times = 2) {
  return static_cast<int64_t>(l.args.batch) * l.max_seqlen_q > times * static_cast<int64_t>(l.total_q);
}

constexpr int kSms = 148;

// Groups of g query tiles that hold rows of a sequence, over all heads, as far as the lengths on the host tell: all of them where every
// sequence is as long as announced, else the rows' share and half a group at the end of each sequence.
inline bool even_batch(const FwdLaunch& l) { return static_cast<int64_t>(l.args.batch) * l.max_seqlen_q <= l.total_q; }
inline int64_t groups_with_rows(const FwdLaunch& l, int g) {
  const int64_t rows = g * kBlockM, all = (l.max_seqlen_q + rows - 1) / rows * l.args.batch;
  const int64_t some = l.total_q / rows + (l.args.batch + 1) / 2;
  return (even_batch(l) || some > all ? all : some) * l.args.heads;
}

// Blocks that start at once
template <int G>
constexpr int kSlots = (G == 1 ? 2 : 1) * kSms;

// Causal grids with their last tiles in order of weight (set_tail_grid): where the blocks do not all start at once, and not up to 512
// queries (four tiles: nothing to gain, and with a CTA per block a place that is computed cost 5-8 %).
inline bool tail_order(const FwdLaunch& l) { return l.max_seqlen_q > 512; }

// Whether a CTA goes on with blocks that have not started (cluster launch control, in the order of the grid) where there are more
// than start at once.  The next block's Q, K and V load and its first scores are made while the rows of the one before leave; a CTA
// of its own began with barriers, tensor memory and 3500 clk for its first scores, about two key tiles.  us, a CTA per block -> now:
// d = 128, 16 x 12 x 1000 causal 85.5 -> 77.7, 64 x 12 x 256 59.4 -> 49.1, 32 x 12 x 512 ragged 61.4 -> 54.7, in pairs of tiles 4 x 32 x
// 3000 causal 293 -> 269, 4 x 12 x 4096 343 -> 328, 16 x 12 x 8192 causal 2570 -> 2490; d = 64, 64 x 12 x 300 69.7 -> 59.3, padded
// 64 x 12 x 512 ragged 92 -> 82; blocks without queries, which the producer passes over: 1 x 4096 and 63 x 128 tokens, 12 heads 182 ->
// 116 (d = 64), 172 -> 128.
// Quads of d = 64 up to some length alone: their two CTAs on an SM take longer for a tile, most of all in long walks (32 768 tokens, 12 heads,
// not causal / causal, over a CTA per block: 600 0.95 / 0.87, 1024 0.96 / 0.92, 1500 0.99 / 0.95, 2048 1.02 / 0.96, 2560 1.01 / 0.99, 3000
// 1.02 / 1.00, 4096 1.08 / 1.02, 1 x 2 x 65536 causal 1.09), unless most blocks are empty (31 x 256 and 1 x 8192: 0.97 / 0.91; announced with 2.5
// times their tokens, 2 x 16384 and 3 x 1, 1.04).  Not with dropout: the loop has no registers left for it (8-14 % slower).
// Nor in grids of few rounds, where little is taken over and a block that was asked for early waits for its CTA while others end.  Time
// over that of a CTA per block, 12 heads, by rounds (announced blocks over those that start at once):
//   quads, not causal    6 x 600 ragged 1.14 (1.2), 5 x 1500 ragged 1.15 (2.4), 14 x 600 1.10 (2.8), 11 x 1000 ragged 1.08 (3.6), 25 x 600 0.94 (5); even
//                        batches 0.96-0.97 up to 1.5
//   quads, causal        7 x 700 1.07 (1.7), 5 x 900 1.09, 9 x 1000 1.03 (2.9), 17 x 600 0.97 (3.4), 11 x 1000 0.98 (3.6), 21 x 700 0.94 (5)
//   rows (d = 64), single tiles (d = 128)   even batches 0.9-0.98 from one round on; where the blocks with rows start at once, 14 x 200 of 1 to 200
//                        tokens 1.19-1.23, 9 x 300 ragged 1.04-1.12
//   d = 128, causal, up to 512 queries (no order of weight)   15 x 300 1.12 (1.8), 18 x 300 ragged 1.15, 17 x 200 of 1 to 200 tokens 1.25; from 3.25
//                        rounds of blocks with rows on 0.94-1.0, even batches of four tiles 1.05 (1.8), 16 x 512 0.96 (2.6)
// Up to 128 queries, and in pairs of query tiles, it pays at any size (0.9, 0.93-0.97 just above one round).
template <int D, bool ROWS, bool CAUSAL>
constexpr int kTakeMaxKeys = D == 64 && !ROWS ? (CAUSAL ? 2560 : 1536) : INT_MAX;
template <int D, int G, bool ROWS, bool CAUSAL>
bool take_over_pays(const FwdLaunch& l, int64_t blocks) {
  if (uneven(l, 3)) return true;
  if (l.max_seqlen_k > kTakeMaxKeys<D, ROWS, CAUSAL>) return false;
  if (l.max_seqlen_q <= kBlockM || (ROWS && G == 2)) return true;
  if (!ROWS) return 4 * blocks > (CAUSAL ? 13 : 16) * kSlots<G> || (!CAUSAL && even_batch(l) && 2 * blocks <= 3 * kSlots<G>);
  const bool even = even_batch(l);
  const int rounds40 = D == 128 && CAUSAL && !tail_order(l) ? (even && l.max_seqlen_q > 3 * kBlockM ? 96 : 130) : even ? 40 : 44;  // in fortieths
  return 40 * groups_with_rows(l, G) > rounds40 * kSlots<G>;
}

template <bool DROPOUT, bool BS>
constexpr bool kCanTake = !BS && !DROPOUT;

template <int D, bool CAUSAL, bool DROPOUT, bool BS, int G, bool ROWS>
Order grid_order(const FwdLaunch& l) {
  const int64_t tiles = (l.max_seqlen_q + G * kBlockM - 1) / (G * kBlockM), blocks = tiles * l.args.heads * l.args.batch;
  if (!linear_grid(tiles, l.args.heads, l.args.batch) || blocks <= kSlots<G>) return kPlain;
  if (kCanTake<DROPOUT, BS> && take_over_pays<D, G, ROWS, CAUSAL>(l, blocks)) return kTake;
  return CAUSAL && tail_order(l) ? kLinear : kPlain;
}

// One query tile per CTA (two CTAs per SM) or two.  What one tile gains lies at the two ends of a CTA's walk over the
// keys, which run under the tiles of the SM's other CTA.  What it loses is a share per key tile: two CTAs each read the K
// and V that a pair reads once, and at d = 128 a single stage holds them.
// Time with one tile / with two, 16 x 16 heads, not causal:
//                        d = 64   dropout d = 64   d = 128   dropout d = 128
//   128 queries, 512 keys     0.75       0.85           0.87       0.78
//   256, 512                  0.88       0.94           1.00       0.87
//   256, 4096                 1.06       1.01           1.16       1.07
//   1024, 1024                0.91       0.92           1.02       0.97
//   1024, 8192                1.03       1.04           1.17       1.09
//   4096, 4096 (4 x 16)       1.00       1.01           1.16       1.08
// so d = 64 takes single tiles at every length (causal calls too: 0.95-0.98).
// d = 128 without dropout, whose CTAs go on with other blocks, so that the ends of a walk count for less (one / two, 12 heads, 16 384
// tokens): not causal 200 tokens 1.08, 300 0.94, 512 1.14, 700 1.11, 1000 1.09, 1100 1.08, 1500 1.14, 1800 1.07, 3000 1.16, ragged 200 0.98,
// 512 1.04, 1000 1.07, 2000 1.11; 16 x 256 queries, 512 and 1024 keys 1.09 and 1.16, 600 and 900 1.10, 2000 and 256 1.07 (see
// pairs_fall_short for the others).  Causal, where the tiles of a pair differ by one in their keys
// (even / ragged): 512 0.90 / 0.85, 1000 0.97 / 0.91, 1300 0.94 / 0.96, 1500 1.03 / 0.96, 1800 0.98 / 0.99, 2000 1.06 / 1.01, 2500 1.06 / 1.02,
// 4096 1.07 / 1.03.
// d = 128 with dropout: up to 1024 keys (causal calls count those up to the longest query) one (2000 queries, 256 keys 171 -> 156, 8 of 4096
// and 512 201 -> 183).  Beyond, causal: 2000 0.96, 4096 1.00, 8192 1.01.  Not causal (8 x 12 / 4 x 16 heads): 1100 0.84 / 0.83,
// 1500 1.00 / 1.03, 2000 0.94 / 0.94, 2500 0.97 / 0.97, 3000 1.04 / 0.97, 4096 1.04 / 1.07 (4 x 12 0.97), 6000 1.05 / 1.02, 8192 1.07 / 1.08, 384
// queries and 2048 keys 0.66 / 1.07, 1100 and 4096 0.87 / 0.79: how the last round of CTAs falls decides, and the rule stays.
// A grid of single tiles that fits one per SM spreads over twice the SMs: 16 heads, 1024 queries, 8192 keys 0.72 (d = 64),
// 0.92 (d = 128), 0.63 and 0.78 with dropout.
// A grid of pairs that fills between half of the SMs and all of them runs in one round either way and reads K and
// V once per pair: 80-140 pairs of 200-4000 queries 1.02-1.13, with dropout 0.99-1.15.
// Up to 128 queries both grids have as many CTAs; with long keys at d = 128 one alone on its SM then wants the second
// stage (16 queries, 4096 keys, one -> two: 96 (batch, head) pairs 69 -> 52 us, 144 pairs 80 -> 58).  From 149 on two
// share an SM: 192 pairs 85 us, 128 with two.
// Uneven batches (see `uneven`) announced with more than 4096 tokens take pairs at d = 64 too, which halves their empty blocks:
// 31 x 256 and 1 x 8192, 12 heads 431 -> 374 us, 2 x 16384 and 126 x 64, 4 heads 948 -> 865.
constexpr int kPairsMaxKeys = 640, kOneTileMaxOdd = 2048, kOneTileMaxD128 = 1024, kOneTileMaxCausal = 1920, kOneTileMaxCausalDropout = 4096;  // keys
constexpr int kOneTileMaxUneven = 4096;  // queries and keys, d = 64

// d = 128, not causal, no dropout, where pairs serve most calls (at any length): the calls that single tiles serve better.  Time with
// pairs over that with one tile, 12 heads:
//   three query tiles, a quarter of whose pairs is empty: 384 queries and 2048 keys 1.03
//   pairs begin a second round and single tiles almost fit one: 15 x 256 1.09, 7 x 450 ragged 1.17, 6 x 640 ragged 1.18, 4 x 1100 ragged 1.28, 15 x
//     150 ragged and 1000 keys 1.13 (18 x 256 1.10; beyond 1.5 rounds of single tiles, 1.25 in ragged batches, 0.86-1.05).  Not where the
//     pairs with rows fit one round (5 x 700 ragged 0.91, 5 x 900 of 1 to 900 tokens 0.93), nor where pairs served the call without
//     blocks being taken over (even numbers of tiles beyond 1024 queries: 2 x 2000 0.84)
//   few keys, and second tiles that are often empty: 43 x 150 of 1 to 150 tokens 1.09, 62 x 150 1.11, 14 x 450 ragged 1.12 (sequences of
//     1000 keys 0.89-1.03)
inline bool pairs_fall_short(const FwdLaunch& l) {
  const int q_tiles = (l.max_seqlen_q + kBlockM - 1) / kBlockM;
  if (q_tiles == 3) return true;
  const int64_t tiles = groups_with_rows(l, 1), pairs = groups_with_rows(l, 2);
  if (100 * pairs <= 92 * kSms && 100 * tiles >= 87 * 2 * pairs) return false;
  const bool few = l.max_seqlen_q <= kOneTileMaxD128 || (q_tiles % 2 != 0 && std::max(l.max_seqlen_q, l.max_seqlen_k) <= kOneTileMaxOdd);
  if (few && 4 * tiles <= (even_batch(l) ? 6 : 5) * kSlots<1>) return true;
  return l.max_seqlen_k <= kPairsMaxKeys && !even_batch(l) &&
         (10 * tiles < 8 * 2 * pairs || (100 * tiles < 89 * 2 * pairs && tiles <= 2 * kSlots<1>));
}

template <int D, bool CAUSAL, bool DROPOUT>
bool one_tile_per_cta(const FwdLaunch& l) {
  const int64_t heads = static_cast<int64_t>(l.args.heads) * l.args.batch;
  const int64_t q_tiles = (l.max_seqlen_q + kBlockM - 1) / kBlockM;
  const int64_t tiles = q_tiles * heads, pairs = (q_tiles + 1) / 2 * heads;
  const int keys = CAUSAL ? std::min(l.max_seqlen_k, l.max_seqlen_q) : l.max_seqlen_k;
  const bool one_round = pairs > kSms / 2 && pairs <= kSms;
  if (l.max_seqlen_q <= kBlockM) return D == 64 || DROPOUT || keys <= kOneTileMaxD128 || pairs > kSms;
  if (one_round) return false;
  if (D == 64) return !(uneven(l) && std::max(l.max_seqlen_q, keys) > kOneTileMaxUneven);
  const bool pairs_at_once = !CAUSAL && !DROPOUT && !pairs_fall_short(l);
  if (l.max_seqlen_q <= kOneTileMaxD128 && (tiles <= kSms || (keys <= kOneTileMaxD128 && !pairs_at_once))) return true;
  if (uneven(l) || pairs_at_once) return false;  // (uneven: twice the empty blocks)
  if (keys <= kOneTileMaxD128) return true;
  if (CAUSAL) return keys <= (DROPOUT ? kOneTileMaxCausalDropout : kOneTileMaxCausal);
  return !DROPOUT || q_tiles % 2 != 0 || l.max_seqlen_q > kOneTileMaxD128;
}

// Rows for d = 128 without dropout, and for d = 64 without dropout up to 512 keys: there the ends of a CTA's
// walk are most of it, and twelve warps take longer through them than eight (quads / rows: 12 heads of 128 queries and
// keys 5.9 / 5.7 us, 16 x 16 heads, 128 queries, 512 keys 12.5 / 11.8, 1024 keys and queries 0.98).
constexpr int kRowsMaxD64 = 512;  // keys

template <int D, bool DROPOUT>
bool rows_layout(const FwdLaunch& l) { return !DROPOUT && (D == 128 || l.max_seqlen_k <= kRowsMaxD64); }

// Backward.  Calls with few query tiles at d = 64: a block's K and V are then a good part of its loads and are waited for at its start, so two
// stages hold them, and two (not three) Q and dO.  Whole backward, us, one stage of K and V -> two: 32 x 12 heads, 256 queries, 500 keys
// 76.3 -> 72.8, 1500 178.4 -> 169.4, with dropout 86.9 -> 84.4 and 209.4 -> 204.8; 128 x 12 x 128 80.9 -> 77.1; 64 x 12 x 512 239 -> 247, 85 x
// 384 212 -> 213, with dropout (ragged) up to 384 261 -> 266.  With a causal mask, 128 x 12 x 256 180.9 -> 171.3, with dropout 192 -> 186, but
// not where keys lie behind the last query, whose blocks store zeros and little else: 32 x 12, 40 queries, 1500 keys 52.2 -> 53.3, with
// dropout (28 bytes of spills) 57.7 -> 62.6, 200 queries 83.5 -> 88.0.
constexpr int kShortQueries = 256;
inline bool short_queries(const BwdLaunch& l) {
  const int q_tiles = (l.args.max_seqlen_q + kBlockM - 1) / kBlockM, k_tiles = (l.args.max_seqlen_k + kBlockN - 1) / kBlockN;
  return l.dpad == 64 && l.args.max_seqlen_q <= kShortQueries && int64_t(k_tiles) * l.args.k.heads * l.args.k.batch > kSms &&
         (!l.is_causal || k_tiles <= q_tiles);
}

}  // namespace fa
