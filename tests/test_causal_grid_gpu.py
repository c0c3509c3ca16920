"""GPU test of the block order of the causal grids: sections of (batch, head) pairs, the first one with what the division
leaves over.  The order may not show: every tile is worked on once, whatever longest length is announced."""
import math

import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,longest", [(64, 20000), (64, 140000), (128, 9000), (128, 70000)])
def test_sections_change_nothing(d, longest):
    """21 pairs: 4 sections of 6 (3 in the first) at the shorter announced length, 21 of one pair at the longer; one section
    at 600 (and the same kernels)."""
    from flash_attn_b200 import flash_attn_cuda as fc
    lens, heads, dtype = [130, 257, 64], 7, torch.bfloat16
    q, k, v, dout, cu, _ = U.make_varlen(lens, lens, heads, d, dtype, seed=d)
    scale = 1.0 / math.sqrt(d)

    def run(n):
        out, lse = fc.fwd(q, k, v, cu, cu, n, n, 0.0, scale, False, True, False, None)
        dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
        fc.bwd(dout, q, k, v, out, lse, dq, dk, dv, cu, cu, n, n, 0.0, scale, False, True, None)
        fc.check_device_status()
        rows = torch.cat([lse[b, :, :m] for b, m in enumerate(lens)], dim=1)
        return out, rows, dk, dv, dq

    assert fc.options.deterministic is False
    fc.options.deterministic = True  # fixes the order in which dQ is summed
    try:
        one, many = run(600), run(longest)
    finally:
        fc.options.deterministic = False
    for a, b in zip(one, many):
        assert torch.equal(a, b)
