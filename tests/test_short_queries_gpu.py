"""GPU tests of the backward for at most 256 queries at d = 64, which holds K and V of two blocks: the same bits as calls of a few
blocks, which hold one."""
import math

import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu

LENS_Q = [256, 0, 1, 129, 128, 64, 255, 127, 200, 17] * 4
LENS_K = [128, 40, 129, 300, 0, 257, 100, 640, 1, 130] * 4


@pytest.mark.parametrize("d,dtype,p_dropout", [(32, torch.float16, 0.0), (64, torch.bfloat16, 0.0), (64, torch.float16, 0.2)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("deterministic", [False, True])
def test_against_a_few_sequences_at_a_time(d, dtype, p_dropout, causal, deterministic):
    from flash_attn_b200 import flash_attn_cuda as fc
    heads, few, scale = 6, 2, 1.0 / math.sqrt(d)   # 40 x 6 x 5 blocks against 10 x 2 x 5
    q, k, v, dout, cu_q, cu_k = U.make_varlen(LENS_Q, LENS_K, heads, d, dtype, seed=d)
    longest_k = max(LENS_K)

    def fwd(q, k, v, mask_heads):
        fc.options.mask_heads = mask_heads
        try:
            return fc.fwd(q, k, v, cu_q, cu_k, 256, longest_k, p_dropout, scale, False, causal, False,
                          torch.Generator(device="cuda").manual_seed(1), return_philox=True)
        finally:
            fc.options.mask_heads = None

    def bwd(q, k, v, dout, out, lse, philox, cq, ck, mask_heads):
        grads = [torch.full_like(t, float("nan")) for t in (q, k, v)]
        fc.options.mask_heads, fc.options.deterministic = mask_heads, deterministic
        try:
            fc.bwd(dout, q, k, v, out, lse, *grads, cq, ck, 256, longest_k, p_dropout, scale, False, causal, None,
                   **({"philox": philox} if p_dropout else {}))
        finally:
            fc.options.mask_heads, fc.options.deterministic = None, False
        fc.check_device_status()
        return grads

    out, lse, *philox = fwd(q, k, v, None)
    philox = tuple(philox[-2:])
    got = bwd(q, k, v, dout, out, lse, philox, cu_q, cu_k, None)
    for h in range(0, heads, few):
        part = [t[:, h:h + few].contiguous() for t in (q, k, v, dout, out)]
        # the first ten sequences: the mask of a sequence depends on its place in the batch and on its head
        cq, ck = cu_q[:11].contiguous(), cu_k[:11].contiguous()
        want = bwd(*part, lse[:10, h:h + few].contiguous(), philox, cq, ck, (heads, h))
        rq, rk = slice(0, int(cq[-1])), slice(0, int(ck[-1]))
        assert torch.equal(got[1][rk, h:h + few], want[1][rk]) and torch.equal(got[2][rk, h:h + few], want[2][rk])
        if deterministic:
            assert torch.equal(got[0][rq, h:h + few], want[0][rq])
        else:   # five fp32 terms at most in another order, and one rounding to the 16-bit type
            eps = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
            torch.testing.assert_close(got[0][rq, h:h + few].float(), want[0][rq].float(), rtol=eps,
                                       atol=5 * 2.0 ** -23 * want[0][rq].float().abs().max().item())
