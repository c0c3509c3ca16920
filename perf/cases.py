"""Workloads of the attention library, each one pass through a public entry point as a user's program calls it.

A case is a dict of plain values:

  entry     which entry point runs: "qkv" (flash_attn_unpadded_qkvpacked_func), "rotary" (RotaryEmbedding.apply_qkv on
            (batch, seqlen, 3, heads, d) and then the packed function), "kv" (flash_attn_unpadded_kvpacked_func), "qkv3"
            (flash_attn_unpadded_func), "module" (FlashAttention with a key padding mask), "sparse"
            (flash_blocksparse_attn_func on a 0/1 layout)
  dtype     "fp16" or "bf16"           dropout   probability        causal, backward   truth values
  batch, heads, d                      ragged    sequence lengths between half and all of the maximum, else all equal
  seqlen    longest sequence (of keys), seqlen_q  longest query sequence where it differs ("kv", "qkv3")
"""
import math
import os
import random
import sys

import torch

_PKG = os.path.abspath("flash-attention_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from flash_attn_b200.flash_attention import FlashAttention  # noqa: E402
from flash_attn_b200.flash_attn_interface import (  # noqa: E402
    flash_attn_unpadded_func, flash_attn_unpadded_kvpacked_func, flash_attn_unpadded_qkvpacked_func)
from flash_attn_b200.flash_blocksparse_attn_interface import flash_blocksparse_attn_func  # noqa: E402
from flash_attn_b200.rotary import RotaryEmbedding  # noqa: E402

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_DENSITY = 0.25  # of a block-sparse layout over 256 x 256-token blocks; the diagonal is always kept


def _case(name, entry, dtype, batch, heads, d, seqlen, *, seqlen_q=0, dropout=0.0, causal=False, backward=False, ragged=False):
    c = {"entry": entry, "dtype": dtype, "batch": batch, "heads": heads, "d": d, "seqlen": seqlen,
         "seqlen_q": seqlen_q or seqlen, "dropout": dropout, "causal": causal, "backward": backward, "ragged": ragged}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one short sentence through an encoder layer at evaluation: the smallest call, all latency
        _case("encoder_one_sentence", "qkv", "fp16", 1, 12, 64, 128),
        # BERT-base-shaped training on packed batches (dropout on), from short to long sequences
        _case("bert_train_128", "qkv", "fp16", 8, 12, 64, 128, dropout=0.1, backward=True, ragged=True),
        _case("bert_train_512", "qkv", "fp16", 8, 12, 64, 512, dropout=0.1, backward=True, ragged=True),
        _case("bert_train_4096", "qkv", "fp16", 8, 12, 64, 4096, dropout=0.1, backward=True, ragged=True),
        # an encoder that serves padded batches: unpad, attention, pad
        _case("encoder_padded_batch", "module", "fp16", 64, 12, 64, 512, ragged=True),
        # causal language model training, head size 128
        _case("lm_train_1000", "qkv", "bf16", 16, 12, 128, 1000, causal=True, backward=True),
        _case("lm_train_8192", "qkv", "bf16", 16, 12, 128, 8192, causal=True, backward=True),
        # prompts of a causal language model with rotary embeddings, forward only
        _case("lm_prefill_3000", "rotary", "bf16", 4, 32, 128, 3000, causal=True),
        # one new token per sequence against its cached keys and values
        _case("lm_decode_4096", "kv", "bf16", 16, 32, 128, 4096, seqlen_q=1, ragged=True),
        # decoder attending to encoder states, separate q, k, v
        _case("cross_train_200_1500", "qkv3", "fp16", 16, 8, 64, 1500, seqlen_q=200, backward=True, ragged=True),
        # block-sparse training, 25 % of the 256 x 256 blocks
        _case("sparse_train_4096", "sparse", "fp16", 4, 16, 64, 4096, dropout=0.1, backward=True),
        # long-context training: the heads one GPU of eight holds
        _case("long_context_train_65536", "qkv", "bf16", 2, 4, 64, 65536, causal=True, backward=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_once(rng):
    kind = rng.choice(("encoder", "bert", "bert", "module", "lm_train", "lm_train", "prefill", "decode", "cross", "sparse", "long"))
    if kind == "encoder":
        return _case("", "qkv", rng.choice(("fp16", "bf16")), _log_int(rng, 1, 32), rng.choice((8, 12, 16)),
                     rng.choice((32, 64, 64, 128)), _log_int(rng, 16, 4096), ragged=rng.random() < 0.5)
    if kind == "bert":
        return _case("", "qkv", "fp16", _log_int(rng, 2, 32), rng.choice((12, 12, 16)), rng.choice((32, 64, 64, 64)),
                     _log_int(rng, 64, 4096), dropout=0.1, backward=True, ragged=True)
    if kind == "module":
        train = rng.random() < 0.5
        return _case("", "module", "fp16", _log_int(rng, 4, 96), 12, 64, _log_int(rng, 64, 1024),
                     dropout=0.1 if train else 0.0, backward=train, ragged=True)
    if kind == "lm_train":
        return _case("", "qkv", "bf16", _log_int(rng, 1, 16), rng.choice((12, 16, 32)), rng.choice((64, 128, 128)),
                     _log_int(rng, 256, 8192), causal=True, backward=True, ragged=rng.random() < 0.25)
    if kind == "prefill":
        return _case("", "rotary", rng.choice(("fp16", "bf16", "bf16")), _log_int(rng, 1, 8), rng.choice((12, 16, 32)),
                     rng.choice((64, 128, 128)), _log_int(rng, 64, 8192), causal=True)
    if kind == "decode":
        return _case("", "kv", rng.choice(("fp16", "bf16")), _log_int(rng, 1, 64), rng.choice((12, 16, 32)),
                     rng.choice((64, 128)), _log_int(rng, 128, 16384), seqlen_q=rng.choice((1, 1, 1, 4)), ragged=True)
    if kind == "cross":
        train = rng.random() < 0.6
        return _case("", "qkv3", rng.choice(("fp16", "bf16")), _log_int(rng, 1, 32), rng.choice((8, 12, 16)),
                     rng.choice((32, 64, 64, 128)), _log_int(rng, 64, 2048), seqlen_q=_log_int(rng, 16, 1024),
                     dropout=rng.choice((0.0, 0.1)) if train else 0.0, backward=train, ragged=True)
    if kind == "sparse":
        train = rng.random() < 0.7
        return _case("", "sparse", "fp16", _log_int(rng, 1, 8), rng.choice((12, 16)), 64, _log_int(rng, 512, 8192),
                     dropout=0.1 if train else 0.0, backward=train)
    return _case("", "qkv", "bf16", rng.choice((1, 2)), rng.choice((2, 4, 8)), 64, _log_int(rng, 8192, 65536),
                 causal=True, backward=rng.random() < 0.75)


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        c = _draw_once(rng)
        # a dropout case takes about twice as long for the same operations
        if work(c)["flops"] * (2 if c["dropout"] else 1) <= most:
            return c


def _lengths(case, longest):
    """Sequence lengths: fixed by the case, so that work() knows them."""
    if not case["ragged"] or longest == 1:
        return [longest] * case["batch"]
    r = random.Random(longest * 1000 + case["batch"])
    return [r.randint(-(-longest // 2), longest) for _ in range(case["batch"])]


def _layout(case):
    """0/1 layout over (16-row query blocks, 256-column key blocks), as lists: seeded 256 x 256 blocks."""
    n = -(-case["seqlen"] // 256)
    r = random.Random(n)
    return [[1 if i == j or r.random() < _DENSITY else 0 for j in range(n)] for i in range(n)]


def _pairs(case):
    """Visible (query, key) pairs of one head, summed over the batch."""
    s = case["seqlen"]
    if case["entry"] == "sparse":
        size = lambda i: min(256, s - 256 * i)  # noqa: E731
        return case["batch"] * sum(size(i) * size(j) for i, row in enumerate(_layout(case)) for j, on in enumerate(row) if on)
    k = _lengths(case, s)
    q = k if case["entry"] in ("qkv", "rotary", "module") else _lengths(case, case["seqlen_q"])
    return sum(a * (a + 1) // 2 if case["causal"] else a * b for a, b in zip(q, k))


def work(case):
    h, d = case["heads"], case["d"]
    tk = sum(_lengths(case, case["seqlen"]))
    own = case["entry"] in ("qkv", "rotary", "module", "sparse")
    tq = tk if own else sum(_lengths(case, case["seqlen_q"]))
    if case["entry"] == "module":  # inputs and outputs are padded
        tk = tq = case["batch"] * case["seqlen"]
    values = (2 * tq + 2 * tk) * h * d                # q, out, k, v
    if case["backward"]:
        values += (2 * tq + 2 * tk) * h * d           # dout, dq, dk, dv
    flops = 4.0 * d * h * _pairs(case) * (3.5 if case["backward"] else 1.0)
    return {"bytes": 2.0 * values, "flops": flops}


def tolerance(case):
    # probabilities, their gradients and the results are rounded to the 16-bit type
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}


def _cu(lengths, device):
    return torch.tensor([0] + lengths, dtype=torch.int32).cumsum(0, dtype=torch.int32).to(device)


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    torch.cuda.manual_seed(seed)  # dropout draws from the default generator
    dtype, h, d = _DTYPES[case["dtype"]], case["heads"], case["d"]
    grad = case["backward"]
    entry = case["entry"]

    def normal(*shape, leaf=True):
        return torch.randn(*shape, generator=g, device=dev, dtype=torch.float32).to(dtype).requires_grad_(grad and leaf)

    k_len = _lengths(case, case["seqlen"])
    tk = sum(k_len)
    st = {"entry": entry, "p": case["dropout"], "causal": case["causal"], "grad": grad, "max_k": max(k_len)}
    if entry == "module":
        s = case["seqlen"]
        st["attn"] = FlashAttention(attention_dropout=case["dropout"]).train(grad)
        st["inputs"] = (normal(case["batch"], s, 3, h, d),)
        st["mask"] = torch.arange(s, device=dev)[None, :] < torch.tensor(k_len, device=dev)[:, None]
        st["dout"] = normal(case["batch"], s, h, d, leaf=False) if grad else None
        return st
    st["cu_k"] = _cu(k_len, dev)
    if entry == "rotary":
        st["inputs"] = (normal(case["batch"], case["seqlen"], 3, h, d),)
        st["rotary"] = RotaryEmbedding(d).to(dev)
    elif entry in ("qkv", "sparse"):
        st["inputs"] = (normal(tk, 3, h, d),)
        st["dout"] = normal(tk, h, d, leaf=False) if grad else None
        if entry == "sparse":
            st["layout"] = torch.tensor(_layout(case), dtype=torch.int32).repeat_interleave(16, dim=0).to(dev)
    else:
        q_len = _lengths(case, case["seqlen_q"])
        tq = sum(q_len)
        st["cu_q"], st["max_q"] = _cu(q_len, dev), max(q_len)
        if entry == "kv":
            st["inputs"] = (normal(tq, h, d), normal(tk, 2, h, d))
        else:
            st["inputs"] = (normal(tq, h, d), normal(tk, h, d), normal(tk, h, d))
        st["dout"] = normal(tq, h, d, leaf=False) if grad else None
    return st


def _forward(st):
    entry, x = st["entry"], st["inputs"]
    if entry == "module":
        return st["attn"](x[0], key_padding_mask=st["mask"], causal=st["causal"])[0]
    if entry == "qkv":
        return flash_attn_unpadded_qkvpacked_func(x[0], st["cu_k"], st["max_k"], st["p"], causal=st["causal"])
    if entry == "rotary":
        b, s, three, h, d = x[0].shape
        qkv = st["rotary"].apply_qkv(x[0]).reshape(b * s, three, h, d)
        return flash_attn_unpadded_qkvpacked_func(qkv, st["cu_k"], st["max_k"], st["p"], causal=st["causal"])
    if entry == "sparse":
        return flash_blocksparse_attn_func(x[0], st["cu_k"], st["layout"], st["p"], st["max_k"], causal=st["causal"])
    f = flash_attn_unpadded_kvpacked_func if entry == "kv" else flash_attn_unpadded_func
    return f(*x, st["cu_q"], st["cu_k"], st["max_q"], st["max_k"], st["p"], causal=st["causal"])


def run(state):
    out = _forward(state)
    if not state["grad"]:
        return [out]
    return [out.detach(), *torch.autograd.grad(out, state["inputs"], state["dout"])]
