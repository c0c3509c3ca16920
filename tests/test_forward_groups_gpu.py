"""GPU tests of the forward with one and with two query tiles per CTA: the same call in a grid that takes one
kernel and in a grid that takes the other must agree, and both stay within the repository's bar of the fp32
oracle.  Lengths at the edges of the 128-row tiles and of pairs of them."""
import math

import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,dtype", [(32, torch.float16), (64, torch.float16), (64, torch.bfloat16), (128, torch.bfloat16)])
@pytest.mark.parametrize("causal", [False, True])
def test_one_tile_and_pairs_of_tiles_agree(d, dtype, causal):
    from flash_attn_b200 import flash_attn_cuda as fc
    heads = 10
    lens_q, lens_k = [128, 127, 129, 255, 256, 257, 5, 384], [128, 300, 129, 120, 256, 513, 40, 385]
    q, k, v, dout, cu_q, cu_k = U.make_varlen(lens_q, lens_k, heads, d, dtype, seed=d)
    scale = 1.0 / math.sqrt(d)

    def run(longest):
        out, lse = fc.fwd(q, k, v, cu_q, cu_k, longest, 513, 0.0, scale, False, causal, False, None)
        fc.check_device_status()
        return out, lse[:, :, :384]

    # 8 x 10 heads: 160 pairs at a maximum of 384 (one tile per CTA); one sequence of 10 heads at a time with
    # its grid padded to 80..148 pairs takes the pairs
    one, lse_one = run(384)
    o32, _, _, _ = U.oracle_cpu(q, k, v, dout, cu_q, cu_k, scale, causal)
    o16, _, _, _ = U.oracle_cpu(q, k, v, dout, cu_q, cu_k, scale, causal, dtype=dtype)
    U.assert_within_2x("one tile", one, o32, o16)
    for b in range(len(lens_q)):
        two, lse_two = fc.fwd(q, k, v, cu_q[b:b + 2].contiguous(), cu_k[b:b + 2].contiguous(), 256 * 9, 513, 0.0, scale,
                              False, causal, False, None)   # 10 x 9 pairs
        rows = slice(int(cu_q[b]), int(cu_q[b + 1]))
        # the same tiles in the same order: the same bits
        assert torch.equal(two[rows], one[rows])
        assert torch.equal(lse_two[0, :, :lens_q[b]], lse_one[b, :, :lens_q[b]])


@pytest.mark.parametrize("d", [64, 128])
def test_dropout_agrees_between_the_two(d):
    from flash_attn_b200 import flash_attn_cuda as fc
    n, heads = 300, 20
    q, k, v, _, cu, _ = U.make_varlen([n], [n], heads, d, torch.float16, seed=1)
    outs = []
    for batch in (1, 2):   # 40 pairs: one tile per CTA; 80: pairs (the second sequence is empty)
        c = torch.tensor([0, n] + [n] * (batch - 1), dtype=torch.int32, device="cuda")
        torch.cuda.manual_seed(3)
        outs.append(fc.fwd(q, k, v, c, c, n, n, 0.25, 0.1, False, False, False, None)[0])
    assert torch.equal(outs[0], outs[1])
