"""CPU test of the rules that choose a kernel for a call, on the functions that the launches use (compiled for the host): query tiles
per CTA, softmax layout and order of the forward's grid, stages of the backward.  The cases are those of the GPU tests that aim at a kernel, and the calls on
either side of a rule's line."""
import math
import os
import random
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash-attention_b200", "csrc")
NVCC = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "fa_rules.h"
template <int D, bool CAUSAL, bool DROPOUT, bool BS>
void forward(const fa::FwdLaunch& l) {
  const bool one = fa::one_tile_per_cta<D, CAUSAL, DROPOUT>(l), rows = fa::rows_layout<D, DROPOUT>(l);
  const fa::Order order = one ? (rows ? fa::grid_order<D, CAUSAL, DROPOUT, BS, 1, true>(l) : fa::grid_order<D, CAUSAL, DROPOUT, BS, 1, false>(l))
                              : (rows ? fa::grid_order<D, CAUSAL, DROPOUT, BS, 2, true>(l) : fa::grid_order<D, CAUSAL, DROPOUT, BS, 2, false>(l));
  printf("%d %s %s\n", one ? 1 : 2, rows ? "rows" : "quads", order == fa::kTake ? "take" : order == fa::kLinear ? "linear" : "plain");
}
template <int D, bool CAUSAL>
void forward(const fa::FwdLaunch& l, bool bs) {
  if constexpr (D == 64)
    if (bs) return l.is_dropout ? forward<D, CAUSAL, true, true>(l) : forward<D, CAUSAL, false, true>(l);
  l.is_dropout ? forward<D, CAUSAL, true, false>(l) : forward<D, CAUSAL, false, false>(l);
}
// the order of grids without a tail in order of weight: pair by pair
bool pair_by_pair() {
  for (int tiles : {1, 2, 3, 17, 128, 2000}) for (int heads : {1, 3, 12}) for (int batch : {1, 5, 33}) {
    fa::KernelArgs a;
    std::memset(&a, 0, sizeof a);
    a.heads = heads; a.batch = batch;
    fa::set_tail_grid(&a, tiles, 0);
    for (int i = 0; i < tiles * heads * batch; ++i) {
      int rank, h, b;
      fa::tail_block(a, i, rank, h, b);
      if (rank != i % tiles || h != i / tiles % heads || b != i / tiles / heads) return false;
    }
  }
  return true;
}
int main(int argc, char**) {
  if (argc > 1) return pair_by_pair() ? 0 : 1;
  char kind;
  int d, batch, heads, mq, mk, total, causal, dropout, bs;
  while (scanf(" %c %d %d %d %d %d %d %d %d %d", &kind, &d, &batch, &heads, &mq, &mk, &total, &causal, &dropout, &bs) == 10) {
    if (kind == 'b') {
      fa::BwdLaunch w;
      std::memset(&w, 0, sizeof w);
      w.dpad = d; w.is_causal = causal; w.is_dropout = dropout;
      w.args.k.batch = batch; w.args.k.heads = heads; w.args.max_seqlen_q = mq; w.args.max_seqlen_k = mk;
      puts(fa::short_queries(w) ? "short" : "long");
      continue;
    }
    fa::FwdLaunch l;
    std::memset(&l, 0, sizeof l);
    l.args.batch = batch; l.args.heads = heads;
    l.max_seqlen_q = mq; l.max_seqlen_k = mk; l.total_q = total;
    l.is_dropout = dropout;
    if (d == 64) causal ? forward<64, true>(l, bs) : forward<64, false>(l, bs);
    else causal ? forward<128, true>(l, bs) : forward<128, false>(l, bs);
  }
  return 0;
}
"""


def call(d, q_lens, heads, max_k=None, causal=False, dropout=False, sparse=False, max_q=None):
    """(d is the padded head size, 64 or 128)"""
    max_q = max_q or max(q_lens)
    return ("f", d, len(q_lens), heads, max_q, max_k or max_q, sum(q_lens), int(causal), int(dropout), int(sparse))


# d = 128, one query tile per CTA (the GPU test of these compares each with 64 bits)
SINGLE_TILES_D128 = [([1920, 1300, 1024], 16, None, True), ([1300] * 4 + [700], 12, None, True), ([1921, 900] * 3, 2, None, True),
                     ([300, 384] * 8, 20, [2048, 1900] * 8, False), ([384, 257, 300] * 8, 10, [384, 1, 129] * 8, False)]
# d = 128, both sides of the causal limit of 1920 keys: the same sequences announced with 1920 and with 1921 tokens
LIMIT_D128 = ([1900, 1700, 1919, 1601], 12)
# forwards that take blocks over
TAKE_OVER = [(128, [1000] * 40, 12, False, 2), (128, [300, 256] * 60, 8, True, 1), (64, [300, 512] * 40, 12, False, 1), (64, [1000, 700] * 30, 12, True, 1)]

def backward(d, batch, heads, max_q, max_k, causal=False, dropout=False):
    return ("b", d, batch, heads, max_q, max_k, batch * max_q, int(causal), int(dropout), 0)


CASES = (
    [(call(128, q, h, max(k or q), c), ("1", "rows")) for q, h, k, c in SINGLE_TILES_D128[:2] + SINGLE_TILES_D128[3:]]
    + [(call(128, LIMIT_D128[0], LIMIT_D128[1], n, True, max_q=n), (tiles, "rows")) for n, tiles in ((1920, "1"), (1921, "2"))]
    + [(call(d, q, h, None, c), (str(g), "rows" if d == 128 or max(q) <= 512 else "quads", "take")) for d, q, h, c, g in TAKE_OVER]
    # up to one round of blocks: as they come; causal ones beyond in order of weight; dropout and block-sparse calls never take over
    + [(call(64, [700] * 4, 12), ("2", "quads", "plain")), (call(64, [700] * 2, 12), ("1", "quads", "plain")), (call(64, [1000] * 40, 12, dropout=True), ("1", "quads", "plain")),
       (call(64, [1000] * 40, 12, causal=True, dropout=True), ("1", "quads", "linear")),
       (call(64, [4096] * 4, 16, causal=True, sparse=True), ("1", "quads", "linear")),
       (call(64, [4096] * 8, 12, causal=True), ("1", "quads", "linear")), (call(64, [4096] * 8, 12), ("1", "quads", "plain")),
       (call(128, [4096] * 8, 12, dropout=True), ("1", "quads", "plain"))]
    # grids of few rounds: a CTA per block
    + [(call(64, [600, 450, 300, 560, 420, 330], 12), ("1", "quads", "plain")), (call(64, [600] * 12, 12), ("1", "quads", "plain")),
       (call(64, [600] * 5, 12), ("1", "quads", "take")), (call(64, [600] * 25, 12), ("1", "quads", "take")),
       (call(64, [900] * 5, 12, causal=True), ("1", "quads", "linear")), (call(64, [700] * 21, 12, causal=True), ("1", "quads", "take")),
       (call(64, [200] + [100] * 13, 12), ("1", "rows", "plain")), (call(64, [200] * 14, 12), ("1", "rows", "take")),
       (call(128, [300] * 16, 12, causal=True), ("1", "rows", "plain")), (call(128, [512] * 16, 12, causal=True), ("1", "rows", "take")),
       (call(128, [512] * 11, 12, causal=True), ("1", "rows", "plain")), (call(128, [300] * 41, 12, causal=True), ("1", "rows", "take")),
       (call(128, [700] * 7, 12, causal=True), ("1", "rows", "take")), (call(128, [700] + [300] * 5, 12, causal=True), ("1", "rows", "linear")),
       (call(64, [128] * 30, 12), ("1", "rows", "take")), (call(64, [8192] + [256] * 31, 12), ("2", "quads", "take"))]
    # d = 128, not causal: pairs, but not where they need a second round that single tiles do not, or are half empty
    + [(call(128, [256] * 15, 12), ("1", "rows")), (call(128, [256] * 22, 12), ("2", "rows")), (call(128, [640, 400, 500, 350, 480, 540], 12), ("1", "rows")),
       (call(128, [1100, 570, 630, 730], 12), ("1", "rows")), (call(128, [1100] * 8, 12), ("2", "rows")), (call(128, [2000, 900], 12), ("2", "rows")),
       (call(128, [374, 406, 386, 631, 465], 12, max_q=700), ("2", "rows")), (call(128, [150] + [60, 90] * 21, 12), ("1", "rows")),
       (call(128, [150] + [60, 90] * 21, 12, max_k=1000), ("2", "rows")), (call(128, [512] * 40, 12), ("2", "rows")),
       (call(128, [384] * 40, 12), ("1", "rows")), (call(128, [5000] + [700] * 30, 12), ("2", "rows"))]
    # two stages of K and V in the backward: not with a causal mask and keys that no query sees
    + [(backward(64, 16, 8, 200, 1500), ("short",)), (backward(64, 16, 8, 257, 1500), ("long",)), (backward(64, 32, 12, 40, 1500, dropout=True), ("short",)),
       (backward(64, 12, 12, 200, 128), ("long",)), (backward(64, 64, 12, 256, 256, causal=True), ("short",)),
       (backward(64, 64, 12, 128, 128, causal=True, dropout=True), ("short",)), (backward(64, 32, 12, 40, 1500, causal=True, dropout=True), ("long",)),
       (backward(64, 32, 12, 200, 500, causal=True), ("long",)), (backward(64, 32, 12, 200, 257, causal=True), ("long",)),
       (backward(128, 16, 8, 200, 1500), ("long",))])


@pytest.fixture(scope="module")
def routes(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("needs nvcc")
    tmp = tmp_path_factory.mktemp("routes")
    src, exe = tmp / "routes.cu", tmp / "routes"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-I" + CSRC, str(src), "-o", str(exe)], check=True,
                   capture_output=True, timeout=300)

    def ask(calls, *flags):
        text = "\n".join(" ".join(map(str, c)) for c in calls)
        out = subprocess.run([str(exe), *flags], input=text, capture_output=True, text=True, check=True, timeout=60).stdout
        return [tuple(line.split()) for line in out.splitlines()]

    return ask


def test_routes(routes):
    got = routes([c for c, _ in CASES])
    for (c, want), have in zip(CASES, got):
        assert have[:len(want)] == want, (c, want, have)


def test_order_without_a_tail(routes):
    routes([], "pair_by_pair")


def test_kernels_that_no_call_reaches(routes):
    """The launches leave out: in padded batches (all rows are there) at d = 64 pairs in more than one round; in order of weight without taking
    over, pairs in rows, and padded batches in rows."""
    rng = random.Random(1)

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    calls = []
    for _ in range(20000):
        batch, heads, longest = log_int(1, 4000), rng.choice((1, 2, 4, 12, 16, 32)), log_int(1, 70000)
        total = batch * longest if rng.random() < 0.5 else max(1, int(batch * longest * rng.random()))
        max_k = longest if rng.random() < 0.7 else log_int(1, 70000)
        calls.append(("f", rng.choice((64, 128)), batch, heads, longest, max_k, total, rng.randint(0, 1), 0, 0))
    got = routes(calls)
    for c, (tiles, layout, order) in zip(calls, got):
        padded = c[6] == c[2] * c[4] and c[4] == c[5]
        assert not (padded and c[1] == 64 and tiles == "2" and order != "plain"), c
        assert not (layout == "rows" and order == "linear" and (tiles == "2" or padded)), c
    assert {g[0] for g in got} == {"1", "2"} and {g[2] for g in got} == {"plain", "linear", "take"}
