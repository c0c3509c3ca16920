"""GPU tests of the block-sparse kernels' lists of visited tiles: more than 32 tiles (a ballot each), none, key blocks that nobody
visits, and in the backward the lists that a CTA makes for the blocks it takes over."""
import math

import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu


def _layout(longest, density, seed, empty):
    n = -(-longest // 256)
    g = torch.Generator().manual_seed(seed)
    layout = torch.rand(-(-longest // 16), n, generator=g) < density
    for i in range(n):
        layout[16 * i, i] = True     # (a row block without any key block is left to the other tests)
    if empty:
        layout[:, n // 2] = False    # a key block that no row visits
    return layout.int().cuda()


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("p_dropout", [0.0, 0.2])
@pytest.mark.parametrize("lens,heads,density", [([129, 0, 1, 700, 128, 300, 512, 257] * 4, 6, 0.1), ([4400, 33, 0, 4097], 4, 0.05)])
def test_blocks_taken_over_against_a_cta_each(lens, heads, density, causal, p_dropout):
    """The deterministic mode launches a CTA per block, whose list the whole CTA makes: the same tiles in the same order."""
    from flash_attn_b200 import flash_attn_cuda as fc
    from flash_attn_b200.flash_blocksparse_attn_interface import convert_blockmask
    longest, scale = max(lens), 0.125
    mask = convert_blockmask(_layout(longest, density, 3, empty=True), causal)
    q, k, v, dout, cu, _ = U.make_varlen(lens, lens, heads, 64, torch.float16, seed=1)
    out, lse, *philox = fc.fwd_block(q, k, v, cu, cu, mask, longest, longest, p_dropout, scale, causal, False, None, return_philox=True)

    def run(deterministic):
        grads = [torch.full_like(t, float("nan")) for t in (q, k, v)]
        fc.options.deterministic = deterministic
        try:
            fc.bwd_block(dout, q, k, v, out, lse, *grads, cu, cu, mask, longest, longest, p_dropout, scale, causal, None,
                         **({"philox": tuple(philox[-2:])} if p_dropout else {}))
        finally:
            fc.options.deterministic = False
        fc.check_device_status()
        return grads

    want, got = run(True), run(False)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # dq: fp32 sums of 35 terms at most in another order, each step 2^-24 of the partial sum, and one rounding to 11 bits
    torch.testing.assert_close(got[0].float(), want[0].float(), rtol=2.0 ** -10, atol=35 * 2.0 ** -23 * want[0].float().abs().max().item())


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("longest", [4224, 5000])
def test_forward_beyond_32_tiles(longest, causal):
    """Against 64 bits.  Two query tiles per CTA (uneven batch, beyond 4096) and one."""
    from flash_attn_b200 import flash_attn_cuda as fc
    from flash_attn_b200.flash_blocksparse_attn_interface import convert_blockmask
    layout = _layout(longest, 0.1, 5, empty=False)
    mask = convert_blockmask(layout, causal)
    for lens in ([longest], [longest, 3, 1]):
        q, k, v, _, cu, _ = U.make_varlen(lens, lens, 2, 64, torch.float16, seed=2)
        out = fc.fwd_block(q, k, v, cu, cu, mask, longest, longest, 0.0, 0.125, causal, False, None)[0]
        fc.check_device_status()
        on = layout.bool().repeat_interleave(16, 0)[:longest].repeat_interleave(256, 1)[:, :longest]
        if causal:
            on = on & torch.ones_like(on).tril()
        s = torch.einsum("qhd,khd->hqk", q[:longest].double(), k[:longest].double()) * 0.125
        s = s.masked_fill(~on, float("-inf"))
        want = torch.einsum("hqk,khd->qhd", torch.nan_to_num(s.softmax(-1)), v[:longest].double())
        # P and the result are rounded to 11 bits: 2^-11 max|v| each
        assert (out[:longest].double() - want).abs().max().item() <= 2.0 ** -10 * v.float().abs().max().item()
        assert math.isfinite(out.float().sum().item())
