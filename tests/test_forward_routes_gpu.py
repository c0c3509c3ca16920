"""GPU tests of forwards that take the routes of tests/test_routes_cpu.py: single query tiles at d = 128, both sides of the rules between
single tiles and pairs, blocks taken over into outputs that held NaN, and a launch that fails while its CTAs take blocks over."""
import ctypes
import math
import time

import pytest
import torch

from tests import _util as U
from tests.test_abandoned_wait_gpu import run_out
from tests.test_routes_cpu import LIMIT_D128, SINGLE_TILES_D128

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q_len,heads,k_len,causal", SINGLE_TILES_D128)
def test_single_tiles_against_64_bits(q_len, heads, k_len, causal):
    from flash_attn_b200 import flash_attn_cuda as fc
    k_len = k_len or q_len
    q, k, v, _, cu_q, cu_k = U.make_varlen(q_len, k_len, heads, 128, torch.float16, seed=sum(q_len))
    out = fc.fwd(q, k, v, cu_q, cu_k, max(q_len), max(k_len), 0.0, 128 ** -0.5, False, causal, False, None)[0]
    fc.check_device_status()
    for b in range(len(q_len)):
        qs, ks = slice(int(cu_q[b]), int(cu_q[b + 1])), slice(int(cu_k[b]), int(cu_k[b + 1]))
        s = torch.einsum("qhd,khd->hqk", q[qs].double(), k[ks].double()) * 128 ** -0.5
        if causal:
            s = s.masked_fill(torch.ones_like(s[0], dtype=torch.bool).triu(1), float("-inf"))
        want = torch.einsum("hqk,khd->qhd", s.softmax(-1), v[ks].double())
        # P and the result are rounded to 11 bits: 2^-11 max|v| each
        assert float((out[qs].double() - want).abs().max()) <= 2 ** -10 * float(v.abs().max())


def test_both_sides_of_the_causal_limit_agree():
    """Announced with 1920 tokens (one query tile per CTA) and with 1921 (pairs): the same tiles in the same order, the same bits."""
    from flash_attn_b200 import flash_attn_cuda as fc
    lens, heads = LIMIT_D128
    q, k, v, _, cu, _ = U.make_varlen(lens, lens, heads, 128, torch.bfloat16, seed=1)
    one, two = [fc.fwd(q, k, v, cu, cu, n, n, 0.0, 0.1, False, True, False, None) for n in (1920, 1921)]
    fc.check_device_status()
    assert torch.equal(one[0], two[0])
    for b, n in enumerate(lens):
        assert torch.equal(one[1][b, :, :n], two[1][b, :, :n])


@pytest.mark.parametrize("lens", [[300, 290, 384, 129], [1000, 640, 513, 1]])
def test_many_blocks_and_one_round_agree(lens):
    """d = 128, not causal: pairs and single tiles by the size of the grid (ten times the four sequences, and four of them)."""
    from flash_attn_b200 import flash_attn_cuda as fc
    heads, longest = 12, max(lens)
    q, k, v, _, cu, _ = U.make_varlen(lens * 10, lens * 10, heads, 128, torch.float16, seed=2)
    out, lse = fc.fwd(q, k, v, cu, cu, longest, longest, 0.0, 0.1, False, False, False, None)
    for first in (0, 36):
        part = cu[first:first + 5].contiguous()
        o, s = fc.fwd(q, k, v, part, part, longest, longest, 0.0, 0.1, False, False, False, None)
        fc.check_device_status()
        rows = slice(int(part[0]), int(part[-1]))
        assert torch.equal(out[rows], o[rows])
        for i, n in enumerate(lens):
            assert torch.equal(lse[first + i, :, :n], s[i, :, :n])


def _call(q, k, v, out, lse, cu_q, cu_k, max_q, max_k, scale, causal):
    from flash_attn_b200 import _lib, flash_attn_cuda as fc
    prm = fc._make_fwd((cu_q.numel() - 1, q.shape[0], k.shape[0], q.shape[1], q.shape[2]), q, k, v, out, lse, cu_q, cu_k, max_q, max_k,
                       0.0, scale, causal, 0, 0)
    _lib.check(_lib.lib.fa_fwd(ctypes.byref(prm), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))


# rows, quads, pairs of uneven batches (d = 64); single tiles and pairs (d = 128)
@pytest.mark.parametrize("d,announced", [(64, 384), (64, 700), (64, 5000), (128, 384), (128, 900), (128, 5000)])
@pytest.mark.parametrize("causal", [False, True])
def test_every_row_of_blocks_taken_over(d, announced, causal):
    """Output and statistics held NaN; each sequence as in a call of its own, which starts all its blocks at once."""
    from flash_attn_b200 import flash_attn_cuda as fc
    lens_q = [128, 0, 1, 300, 129, 64, 384, 127, 256, 33] * 12
    lens_k = [128, 40, 129, 300, 0, 257, 100, 384, 1, 130] * 12
    heads, scale = 6, 1.0 / math.sqrt(d)
    q, k, v, _, cu_q, cu_k = U.make_varlen(lens_q, lens_k, heads, d, torch.float16, seed=d)
    out, lse = torch.full_like(q, float("nan")), torch.full((len(lens_q), heads, (announced + 15) // 16 * 16), float("nan"), device="cuda")
    _call(q, k, v, out, lse, cu_q, cu_k, announced, announced, scale, causal)
    fc.check_device_status()
    for b, n in enumerate(lens_q):
        o, s = fc.fwd(q, k, v, cu_q[b:b + 2].contiguous(), cu_k[b:b + 2].contiguous(), announced, announced, 0.0, scale, False, causal,
                      False, None)
        rows = slice(int(cu_q[b]), int(cu_q[b + 1]))
        assert torch.equal(out[rows], o[rows])
        assert torch.equal(lse[b, :, :n], s[0, :, :n])
        assert torch.isnan(lse[b, :, n:]).all()


def _serial():
    """The number of the latest call; those that follow count on."""
    from flash_attn_b200 import flash_attn_cuda as fc
    fc.check_device_status()
    serial = run_out(64, False)[0]
    with pytest.raises(RuntimeError):
        fc.check_device_status()
    return serial


@pytest.mark.parametrize("d,tokens,batch,heads", [(16, 512, 4096, 32), (16, 1024, 1024, 32), (128, 32768, 4, 32)])
def test_blocks_taken_over_do_not_start_after_a_failure(d, tokens, batch, heads):
    """The status word of a launch that is under way (25 ms and more) is set from another stream, as one of its CTAs would set it: blocks that
    have not started stay out, those that were written are right.  Rows, quads, pairs of tiles at d = 128."""
    from flash_attn_b200 import flash_attn_cuda as fc
    x = torch.randn(tokens * batch, heads, d, device="cuda", dtype=torch.float16)
    out, lse = torch.empty_like(x), torch.empty(batch, heads, tokens, device="cuda")
    cu = torch.arange(0, tokens * batch + 1, tokens, dtype=torch.int32, device="cuda")
    status, side, started = fc._status_buffer(x.device), torch.cuda.Stream(), torch.cuda.Event()

    def run():
        _call(x, x, x, out, lse, cu, cu, tokens, tokens, 0.25, False)

    run()
    torch.cuda.synchronize()
    want = out.clone()
    word = torch.tensor([_serial() + 1], dtype=torch.int32).pin_memory()
    status.zero_()
    out.fill_(float("nan"))
    torch.cuda.synchronize()
    started.record()
    run()
    started.synchronize()
    time.sleep(0.004)
    with torch.cuda.stream(side):
        status[:1].copy_(word, non_blocking=True)
    torch.cuda.synchronize()
    missing = torch.isnan(out[:, :, 0])
    assert 0.05 < missing.float().mean().item() < 1.0
    assert torch.equal(out[~missing], want[~missing])
    status.zero_()
    run()
    fc.check_device_status()
    assert torch.equal(out, want)


@pytest.mark.parametrize("d,lens,causal", [(64, [1000, 700, 1, 1000] * 10, False), (64, [1000, 700, 1, 1000] * 10, True), (64, [300, 512] * 40, False),
                                           (128, [1000, 700, 1, 1000] * 10, False), (128, [300, 256] * 60, True)])
def test_a_forward_that_has_failed_takes_nothing_over(d, lens, causal):
    """The word is set before the launch: what was written all the same is right, and the call after it gives what it gave before."""
    from flash_attn_b200 import flash_attn_cuda as fc
    heads, longest = 12, max(lens)
    q, k, v, _, cu, _ = U.make_varlen(lens, lens, heads, d, torch.float16, seed=d)
    out, lse = torch.empty_like(q), torch.empty(len(lens), heads, (longest + 15) // 16 * 16, device="cuda")
    status = fc._status_buffer(q.device)

    def run():
        _call(q, k, v, out, lse, cu, cu, longest, longest, 0.125, causal)
        torch.cuda.synchronize()
        return out.clone()

    want = run()
    serial = _serial()
    out.fill_(float("nan"))
    status[0] = serial + 1
    got = run()
    assert torch.all(torch.isnan(got) | (got == want))
    if longest > 512 and d == 64:   # quads
        assert torch.isnan(got).all()
    status.zero_()
    assert torch.equal(run(), want)
    fc.check_device_status()


@pytest.mark.parametrize("seqlen,d", [(300, 64), (700, 64), (300, 128), (1000, 128)])
def test_a_padded_batch_after_one_that_has_failed(seqlen, d):
    from flash_attn_b200 import flash_attn_cuda as fc
    batch, heads = 60, 6
    x = torch.randn(batch, seqlen, 3, heads, d, device="cuda").half()
    lens = torch.randint(0, seqlen + 1, (batch,), generator=torch.Generator().manual_seed(1))
    mask = (torch.arange(seqlen)[None, :] < lens[:, None]).cuda()
    native = fc.compiled_attention(x)
    want = native.attn_padded_qkv(x, mask, None, False)
    serial, status = _serial(), fc._status_buffer(x.device)
    status[0] = serial + 1
    native.attn_padded_qkv(x, mask, None, False)
    torch.cuda.synchronize()
    status.zero_()
    assert torch.equal(native.attn_padded_qkv(x, mask, None, False), want)
    fc.check_device_status()
