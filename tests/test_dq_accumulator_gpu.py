"""GPU tests of the two layouts of the fp32 dQ accumulator (one block per query tile up to 512 tokens and with
dropout, boxes of rows beyond): sequences that start at any row, end inside a tile and at the end of the tensor.  Bar: the repository's 2x rule against the fp32 oracle."""
import math

import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [16, 64])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("lens_q,lens_k", [([512, 37, 300], [512, 200, 129]), ([3, 130, 129], [400, 5, 640]), ([511], [385])])
def test_both_layouts_against_the_oracle(d, causal, lens_q, lens_k):
    from flash_attn_b200 import flash_attn_cuda as fc
    q, k, v, dout, cu_q, cu_k = U.make_varlen(lens_q, lens_k, 3, d, torch.float16, seed=d + len(lens_q))
    scale = 1.0 / math.sqrt(d)
    _, *want = U.oracle_cpu(q, k, v, dout, cu_q, cu_k, scale, causal)
    _, *lowp = U.oracle_cpu(q, k, v, dout, cu_q, cu_k, scale, causal, dtype=torch.float16)
    for longest in (512, 1024):
        out, lse = fc.fwd(q, k, v, cu_q, cu_k, longest, max(lens_k), 0.0, scale, False, causal, False, None)
        grads = [torch.full_like(x, float("nan")) for x in (q, k, v)]
        fc.bwd(dout, q, k, v, out, lse, *grads, cu_q, cu_k, longest, max(lens_k), 0.0, scale, False, causal, None)
        fc.check_device_status()
        for name, got, w, l in zip(("dq", "dk", "dv"), grads, want, lowp):
            U.assert_within_2x(name, got, w, l)
