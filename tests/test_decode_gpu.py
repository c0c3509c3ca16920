"""GPU tests of the forward kernel for one to four query rows per sequence, against the fp32 CPU oracle.

Bar: max|x - ref32| <= 2 * max|lowp - ref32| + 1e-4 (the repository's rule), LSE within 2e-4."""
import math

import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu


# key counts at the edges of a CTA's unit (8 warps x 64 / (d / 8) .. keys) and of the split rule (256 keys
# per CTA and doubling); several heads and sequences change the number of splits
@pytest.mark.parametrize("d,dtype", [(16, torch.float16), (32, torch.bfloat16), (64, torch.float16),
                                     (64, torch.bfloat16), (128, torch.float16), (128, torch.bfloat16)])
@pytest.mark.parametrize("sq,sk,heads", [
    ([1], [1], 2), ([1, 1, 1], [127, 128, 129], 3), ([1, 1], [511, 512], 1), ([1], [1025], 2),
    ([1, 1], [0, 300], 2), ([0, 1, 1], [5, 2047, 4100], 1), ([1] * 40, [600] * 39 + [17], 16),
    ([4], [255], 2), ([4, 1, 3, 0, 2], [1, 64, 257, 33, 1100], 2), ([2, 4], [2049, 1], 3),
])
def test_few_query_rows(d, dtype, sq, sk, heads):
    from flash_attn_b200 import flash_attn_cuda as fc
    q, k, v, dout, cu_q, cu_k = U.make_varlen(sq, sk, heads, d, dtype, seed=len(sq) + d)
    kv = torch.stack([k, v], dim=1)  # packed cache: strided views
    scale = 1.0 / math.sqrt(d)
    # rows outside every sequence and LSE entries of absent rows keep what was there
    out, lse = fc.fwd(q, kv[:, 0], kv[:, 1], cu_q, cu_k, max(sq), max(max(sk), 1), 0.0, scale, False, False, False, None)
    torch.cuda.synchronize()
    fc.check_device_status()
    o32, _, _, _ = U.oracle_cpu(q, k, v, dout, cu_q, cu_k, scale, False)
    o16, _, _, _ = U.oracle_cpu(q, k, v, dout, cu_q, cu_k, scale, False, dtype=dtype)
    lses = U.oracle_lse(q, k, v, cu_q, cu_k, scale, False)
    start = 0
    for b, (n, m) in enumerate(zip(sq, sk)):
        rows = slice(start, start + n)
        start += n
        if n == 0:
            continue
        if m == 0:  # no key: zeros and -inf
            assert (out[rows] == 0).all() and torch.isneginf(lse[b, :, :n]).all()
            continue
        U.assert_within_2x("out", out[rows], o32[rows], o16[rows])
        assert U.max_err(lse[b, :, :n], lses[b]) < 2e-4


def test_same_numbers_as_the_tile_kernel():
    """The rows come out of the tile kernel as well when a longer maximum sends the call there.  Both round
    the result to fp16 once (2^-11) and the tile kernel also rounds each probability: 2^-10 of the largest
    value a row can reach."""
    from flash_attn_b200 import flash_attn_cuda as fc
    sq, sk = [1, 3, 2], [700, 64, 1500]
    q, k, v, _, cu_q, cu_k = U.make_varlen(sq, sk, 4, 64, torch.float16, seed=2)
    a, lse_a = fc.fwd(q, k, v, cu_q, cu_k, 4, 1500, 0.0, 0.125, False, False, False, None)
    b, lse_b = fc.fwd(q, k, v, cu_q, cu_k, 16, 1500, 0.0, 0.125, False, False, False, None)
    assert U.max_err(a, b) <= 2 ** -10 * v.float().abs().max().item()
    for i, n in enumerate(sq):
        assert U.max_err(lse_a[i, :, :n], lse_b[i, :, :n]) < 2e-4


def test_keys_outside_the_tensor_read_as_zero():
    """cu_seqlens past the end of the key tensor: the missing rows count as zero keys and values, as in the
    tile kernel, and are not read."""
    from flash_attn_b200 import flash_attn_cuda as fc
    q, k, v, _, cu_q, _ = U.make_varlen([1], [100], 2, 64, torch.float16, seed=5)
    cu_k = torch.tensor([0, 130], dtype=torch.int32, device="cuda")
    out, _ = fc.fwd(q, k, v, cu_q, cu_k, 1, 130, 0.0, 0.125, False, False, False, None)
    pad = torch.zeros(30, 2, 64, dtype=torch.float16, device="cuda")
    want, _ = fc.fwd(q, torch.cat([k, pad]), torch.cat([v, pad]), cu_q, cu_k, 1, 130, 0.0, 0.125, False, False, False, None)
    assert torch.equal(out, want)


def test_infinite_and_nan_scores():
    """A row whose scores hold +inf or NaN is NaN, as in the tile kernel; -inf scores count nothing."""
    from flash_attn_b200 import flash_attn_cuda as fc
    q, k, v, _, cu_q, cu_k = U.make_varlen([1, 1, 1], [300, 300, 300], 1, 64, torch.float16, seed=6)
    q = q.abs() + 0.1
    k[40, 0, 0] = float("inf")
    k[340, 0, 0] = float("nan")
    k[700, 0, 0] = float("-inf")
    for longest in (1, 16):  # this kernel, the tile kernel
        out, lse = fc.fwd(q, k, v, cu_q, cu_k, longest, 300, 0.0, 0.125, False, False, False, None)
        assert torch.isnan(out[0]).all() and torch.isnan(out[1]).all() and torch.isfinite(out[2]).all()
        assert torch.isneginf(lse[0, 0, 0]) and torch.isneginf(lse[1, 0, 0]) and torch.isfinite(lse[2, 0, 0])


# announced key counts on the two sides of the rule that chooses the kernel: (rows, pairs, d) and the first count
@pytest.mark.parametrize("rows,batch,heads,d,edge", [(1, 30, 4, 64, 1024), (1, 64, 4, 128, 8193), (3, 30, 4, 32, 4097), (2, 8, 4, 128, 512),
                                                     (4, 8, 4, 128, 65), (2, 20, 4, 64, 257), (4, 20, 4, 128, 65)])
def test_both_kernels_at_the_edges_of_the_rule(rows, batch, heads, d, edge):
    """The same sequences through both (tolerance as above)."""
    from flash_attn_b200 import flash_attn_cuda as fc
    keys = [1 + (37 * i) % min(edge - 1, 700) for i in range(batch)]
    q, k, v, _, cu_q, cu_k = U.make_varlen([rows] * batch, keys, heads, d, torch.float16, seed=rows + d)
    runs = [fc.fwd(q, k, v, cu_q, cu_k, rows, longest, 0.0, 0.125, False, False, False, None) for longest in (edge - 1, edge)]
    fc.check_device_status()
    assert U.max_err(runs[0][0], runs[1][0]) <= 2 ** -10 * v.float().abs().max().item()
    assert U.max_err(runs[0][1][:, :, :rows], runs[1][1][:, :, :rows]) < 2e-4
