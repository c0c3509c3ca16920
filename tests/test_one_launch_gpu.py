"""Backward with at most 128 queries and keys per sequence: the main kernel alone (softmax_d and dq written by it) against the three kernels
(all stages asked for by name).  Every dQ tile is one product, so the results are the same bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q_len,k_len,heads,d,dtype,causal,p", [
    ([1], [1], 1, 64, torch.float16, False, 0.0),
    ([128, 128], [128, 128], 2, 64, torch.float16, False, 0.1),
    ([127, 0, 65, 1], [127, 0, 65, 1], 3, 32, torch.float16, True, 0.0),
    ([100, 128, 17], [77, 0, 128], 2, 64, torch.bfloat16, False, 0.1),       # a sequence without keys
    ([100, 5, 128], [100, 128, 3], 2, 128, torch.bfloat16, False, 0.0),
    ([31, 97, 64], [128, 17, 64], 3, 128, torch.float16, True, 0.2),
    ([40] * 9, [90] * 9, 16, 16, torch.float16, False, 0.1),
    ([128, 100, 0, 33] * 9, [128, 60, 7, 0] * 9, 4, 64, torch.float16, False, 0.0),
    ([128, 33, 0, 96] * 4, [128, 33, 0, 120] * 4, 9, 128, torch.bfloat16, True, 0.1)])
def test_main_kernel_alone(q_len, k_len, heads, d, dtype, causal, p):
    from flash_attn_b200 import flash_attn_cuda as fc
    g = torch.Generator(device="cuda").manual_seed(sum(q_len) + d)
    tq, tk, mq, mk = sum(q_len), sum(k_len), max(q_len), max(k_len)
    cu_q, cu_k = (torch.tensor([0] + x, dtype=torch.int32).cumsum(0, dtype=torch.int32).cuda() for x in (q_len, k_len))

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g).to(dtype)

    # two spare rows behind the sequences, which belong to nobody
    q, k, v, dout = normal(tq + 2, heads, d), normal(tk + 2, heads, d), normal(tk + 2, heads, d), normal(tq + 2, heads, d)
    out, lse, seed, offset = fc.fwd(q, k, v, cu_q, cu_k, mq, mk, p, d ** -0.5, False, causal, False, g, return_philox=True)
    got = []
    for stages in (0, 7):
        grads = [torch.full_like(x, 3.0) for x in (q, k, v)]
        sd = fc.bwd(dout, q, k, v, out, lse, *grads, cu_q, cu_k, mq, mk, p, d ** -0.5, False, causal, None,
                    philox=(seed, offset), _stage_mask=stages)[3]
        got.append(grads + [sd])
    fc.check_device_status()
    for a, b in zip(got[0][:3], got[1][:3]):
        assert torch.equal(a, b)
    assert torch.equal(got[0][0][tq:], torch.full_like(q[tq:], 3.0))
    for i, n in enumerate(q_len):
        assert torch.equal(got[0][3][i, :, :n], got[1][3][i, :, :n])


def test_which_calls_need_a_workspace():
    from flash_attn_b200 import _lib
    needs = _lib.lib.fa_bwd_needs_workspace
    assert needs(37, 4, 128, 128, 0, 0) == 0
    assert all(needs(*x) == 1 for x in ((149, 1, 128, 128, 0, 0), (37, 4, 129, 128, 0, 0), (37, 4, 128, 129, 0, 0),
                                        (37, 4, 128, 128, 1, 0), (37, 4, 128, 128, 0, 2)))
