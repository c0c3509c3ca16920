"""GPU tests of the forward's grids with more blocks than start at once, whose CTAs go on with blocks that have not started: the
same tiles in the same order as in grids whose blocks have a CTA each, so the same bits."""
import math

import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu

# tiles without keys, without queries, with one row, at the edges of 128; a row on either side of a warp's 32 rows
LENS_Q = [128, 0, 1, 300, 129, 64, 384, 127, 256, 33] * 5
LENS_K = [128, 40, 129, 300, 0, 257, 100, 384, 1, 130] * 5


# announced lengths and what they choose: rows (d = 64 up to 512 keys, d = 128), quads; one query tile per CTA, or two (uneven
# batches beyond 4096)
@pytest.mark.parametrize("d,dtype,announced", [(32, torch.float16, 384), (64, torch.bfloat16, 384), (64, torch.float16, 700),
                                               (16, torch.bfloat16, 1500), (64, torch.float16, 5000), (128, torch.bfloat16, 384),
                                               (128, torch.float16, 900), (128, torch.bfloat16, 5000)])
@pytest.mark.parametrize("causal", [False, True])
def test_one_launch_and_one_per_sequence_agree(d, dtype, announced, causal):
    from flash_attn_b200 import flash_attn_cuda as fc
    heads, scale = 6, 1.0 / math.sqrt(d)   # 50 x 6 x 3 blocks at least against 6 x 40 at most
    q, k, v, _, cu_q, cu_k = U.make_varlen(LENS_Q, LENS_K, heads, d, dtype, seed=d)

    def run(cq, ck):
        out, lse = fc.fwd(q, k, v, cq, ck, announced, announced, 0.0, scale, False, causal, False, None)
        fc.check_device_status()
        return out, lse

    out, lse = run(cu_q, cu_k)
    for b, n in enumerate(LENS_Q):
        if n == 0 or b >= 20:
            continue
        o, s = run(cu_q[b:b + 2].contiguous(), cu_k[b:b + 2].contiguous())
        rows = slice(int(cu_q[b]), int(cu_q[b + 1]))
        assert torch.equal(out[rows], o[rows])
        assert torch.equal(lse[b, :, :n], s[0, :, :n])
    # the second half of the batch repeats the lengths: every row was written
    assert not torch.isnan(out).any() and not torch.isnan(lse[:, :, :1]).any()
    ref = fc.fwd(q, k, v, cu_q[30:].contiguous(), cu_k[30:].contiguous(), announced, announced, 0.0, scale, False, causal, False, None)[0]
    assert torch.equal(out[int(cu_q[30]):], ref[int(cu_q[30]):])


@pytest.mark.parametrize("batch,seqlen,heads,d,causal", [(40, 300, 6, 64, False), (40, 300, 6, 32, True), (24, 700, 6, 64, False),
                                                         (24, 700, 6, 64, True), (40, 300, 6, 128, False), (30, 1100, 4, 128, True)])
def test_padded_batches(batch, seqlen, heads, d, causal):
    """Blocks without a token are passed on too: their rows get zeros."""
    from flash_attn_b200 import flash_attn_cuda as fc
    g = torch.Generator(device="cuda").manual_seed(seqlen)
    x = torch.randn(batch, seqlen, 3, heads, d, device="cuda", generator=g).half()
    lens = torch.randint(0, seqlen + 1, (batch,), generator=torch.Generator().manual_seed(1))
    lens[0], lens[1], lens[2] = seqlen, 0, 1
    mask = (torch.arange(seqlen)[None, :] < lens[:, None]).cuda()
    x[~mask] = float("nan")
    native = fc.compiled_attention(x)
    torch.full((batch, seqlen, heads, d), float("nan"), dtype=x.dtype, device="cuda")   # (what the output's memory may hold)
    got = native.attn_padded_qkv(x, mask, None, causal)
    for b in range(0, batch, 5):
        one = native.attn_padded_qkv(x[b:b + 1].contiguous(), mask[b:b + 1].contiguous(), None, causal)
        assert torch.equal(got[b], one[0])
    assert torch.all(got[~mask] == 0) and not torch.isnan(got).any()


@pytest.mark.parametrize("d", [64, 128])
def test_captured_and_on_two_streams(d):
    from flash_attn_b200 import flash_attn_cuda as fc
    lens, heads, scale = [300, 17, 512, 256] * 10, 8, 1.0 / math.sqrt(d)
    q, k, v, _, cu, _ = U.make_varlen(lens, lens, heads, d, torch.float16, seed=d)
    call = lambda: fc.fwd(q, k, v, cu, cu, 512, 512, 0.0, scale, False, True, False, None)[0]  # noqa: E731
    want = call()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        out = call()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(3):
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        got = []
        for s in streams:
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                got.append(call())
        torch.cuda.synchronize()
        assert all(torch.equal(o, want) for o in got)
    fc.check_device_status()
