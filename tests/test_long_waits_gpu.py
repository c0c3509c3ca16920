"""GPU tests of waits that span another role's work in kernels whose CTAs go on with blocks that have not started: longer than the limit of
a wait, because the producer passes over some 100 000 blocks without work, or because one group walks a long sequence while the other
group of its CTA has no rows.  The launch is not abandoned, and its results are those of the same sequences in a call without them."""
import math

import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu

LENS = [300, 17, 129, 256]


def _announced(batch):
    """LENS at both ends of `batch` sequences, the others of length zero."""
    return LENS + [0] * (batch - 2 * len(LENS)) + LENS


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_backward_of_sequences_without_keys(d, causal):
    """8192 x 16 x 512 blocks at 0.5 us of an SM each: 0.2 s."""
    from flash_attn_b200 import flash_attn_cuda as fc
    batch, heads, scale = 8192, 16, 1.0 / math.sqrt(d)
    lens = LENS * 2
    q, k, v, dout, cu, _ = U.make_varlen(lens, lens, heads, d, torch.float16, seed=d)
    out, lse = fc.fwd(q, k, v, cu, cu, 300, 300, 0.0, scale, False, causal, False, None)

    def run(cu, stats, longest):
        grads = [torch.full_like(t, float("nan")) for t in (q, k, v)]
        fc.bwd(dout, q, k, v, out, stats, *grads, cu, cu, 300, longest, 0.0, scale, False, causal, None)
        fc.check_device_status()
        return grads

    want = run(cu, lse, 300)
    wide = torch.zeros(batch, heads, lse.shape[2], device="cuda")
    wide[:4], wide[-4:] = lse[:4], lse[4:]
    ends = torch.tensor([0] + _announced(batch)).cumsum(0).int().cuda()
    got = run(ends, wide, 65536)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # dq: three fp32 terms at most in another order, and one rounding to 11 bits
    torch.testing.assert_close(got[0].float(), want[0].float(), rtol=2.0 ** -10, atol=1e-5 * want[0].float().abs().max().item())


def test_block_sparse_backward_of_sequences_without_keys():
    """2048 x 16 x 1024 blocks, whose lists are made for those with keys alone."""
    from flash_attn_b200 import flash_attn_cuda as fc
    from flash_attn_b200.flash_blocksparse_attn_interface import convert_blockmask
    batch, heads, longest = 2048, 16, 131072
    lens = LENS * 2
    q, k, v, dout, cu, _ = U.make_varlen(lens, lens, heads, 64, torch.float16, seed=1)
    layout = torch.ones(32, longest // 256, dtype=torch.int32, device="cuda")
    layout[3, 0], layout[7, 1] = 0, 0
    wide_mask, mask = convert_blockmask(layout, False), convert_blockmask(layout[:, :2].contiguous(), False)
    out, lse = fc.fwd_block(q, k, v, cu, cu, mask, 300, 300, 0.0, 0.125, False, False, None)

    def run(cu, stats, mask, longest):
        grads = [torch.full_like(t, float("nan")) for t in (q, k, v)]
        fc.bwd_block(dout, q, k, v, out, stats, *grads, cu, cu, mask, 300, longest, 0.0, 0.125, False, None)
        fc.check_device_status()
        return grads

    want = run(cu, lse, mask, 300)
    wide = torch.zeros(batch, heads, lse.shape[2], device="cuda")
    wide[:4], wide[-4:] = lse[:4], lse[4:]
    got = run(torch.tensor([0] + _announced(batch)).cumsum(0).int().cuda(), wide, wide_mask, longest)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    torch.testing.assert_close(got[0].float(), want[0].float(), rtol=2.0 ** -10, atol=1e-5 * want[0].float().abs().max().item())


@pytest.mark.parametrize("d", [64, 128])
def test_forward_of_sequences_without_queries(d):
    """8192 x 16 x 256 pairs of tiles; the softmax_lse of the announced lengths takes 34 GB."""
    from flash_attn_b200 import flash_attn_cuda as fc
    batch, heads, longest, scale = 8192, 16, 65536, 1.0 / math.sqrt(d)
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 34 GB of device memory")
    lens = LENS * 2
    q, k, v, dout, cu, _ = U.make_varlen(lens, lens, heads, d, torch.float16, seed=d)
    want = fc.fwd(q, k, v, cu, cu, 300, 300, 0.0, scale, False, False, False, None)[0]
    ends = torch.tensor([0] + _announced(batch)).cumsum(0).int().cuda()
    got = fc.fwd(q, k, v, ends, ends, longest, longest, 0.0, scale, False, False, False, None)[0]
    fc.check_device_status()
    if d == 128:
        assert torch.equal(got, want)
    else:   # quads and rows: sums of 300 fp32 terms in another order, one unit of the output
        torch.testing.assert_close(got.float(), want.float(), rtol=2.0 ** -10, atol=2.0 ** -24)
    torch.cuda.empty_cache()


@pytest.mark.parametrize("d,dtype,keys", [(16, torch.float16, 40_000_000), (128, torch.bfloat16, 16_000_000)])
def test_one_group_walks_while_the_other_has_no_rows(d, dtype, keys):
    """Five query tiles in pairs: the last CTA's second group waits for the next block while the first walks 125 000 key tiles and more, at
    1500 clk at least.  All keys but 600 score below -40 and weigh nothing."""
    from flash_attn_b200 import flash_attn_cuda as fc
    queries, others, scale = 640, 59, 1.0 / math.sqrt(d)
    g = torch.Generator(device="cuda").manual_seed(d)
    q = torch.randn(queries + others, 1, d, device="cuda", generator=g).abs().add_(0.5).to(dtype)
    k, v = (torch.empty(keys + others, 1, d, dtype=dtype, device="cuda") for _ in range(2))
    k.fill_(-64.0 / math.sqrt(d))
    v.fill_(1.0)
    seen = torch.cat([torch.arange(300), torch.arange(keys - 300, keys)]).cuda()
    k[seen] = torch.randn(600, 1, d, device="cuda", generator=g).to(dtype)
    v[seen] = torch.randn(600, 1, d, device="cuda", generator=g).to(dtype)
    cu_q = torch.tensor([0, queries] + [queries + 1 + i for i in range(others)], dtype=torch.int32, device="cuda")
    cu_k = torch.tensor([0, keys] + [keys + 1 + i for i in range(others)], dtype=torch.int32, device="cuda")
    out = fc.fwd(q, k, v, cu_q, cu_k, queries, keys, 0.0, scale, False, False, False, None)[0]
    fc.check_device_status()
    s = q[:queries, 0].double() @ k[seen, 0].double().T * scale
    weight = s.logsumexp(1) - (q[:queries, 0].double().sum(1) * float(k[400, 0, 0]) * scale + math.log(keys))
    assert weight.min() > 16   # the others weigh less than 2^-23 of them
    want = s.softmax(-1) @ v[seen, 0].double()
    # P and the result are rounded to 11 or 8 bits: half a unit of max|v| each
    unit = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert float((out[:queries, 0].double() - want).abs().max()) <= 2 * unit * float(v.abs().max())
    assert torch.equal(out[queries:], v[keys:])
