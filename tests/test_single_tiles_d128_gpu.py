"""d = 128, both sides of the lines between one query tile per CTA and pairs: causal calls of 2560 keys, odd and even numbers of
query tiles, few keys, uneven batches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q_len,k_len,causal", [
    ([2560, 1200], None, True), ([2561, 2000], None, True), ([1100, 900], None, False), ([1200, 1030], None, False),
    ([2048, 2047], None, False), ([1920, 1921], None, False), ([300, 384], [2048, 1900], False), ([300, 384], [2049, 1900], False),
    ([2000, 1500], [256, 1], False), ([2300] + [20] * 7, None, True)])
def test_against_64_bits(q_len, k_len, causal):
    from flash_attn_b200.flash_attn_interface import flash_attn_unpadded_func
    k_len = k_len or q_len
    heads, d = 20, 128
    g = torch.Generator(device="cuda").manual_seed(sum(q_len))
    cu_q, cu_k = (torch.tensor([0] + x, dtype=torch.int32).cumsum(0, dtype=torch.int32).cuda() for x in (q_len, k_len))
    q, k, v = (torch.randn(sum(x), heads, d, device="cuda", generator=g).half() for x in (q_len, k_len, k_len))
    out = flash_attn_unpadded_func(q, k, v, cu_q, cu_k, max(q_len), max(k_len), 0.0, causal=causal)
    for b in range(len(q_len)):
        for h in (0, heads - 1):
            qs, ks = slice(int(cu_q[b]), int(cu_q[b + 1])), slice(int(cu_k[b]), int(cu_k[b + 1]))
            s = q[qs, h].double() @ k[ks, h].double().T * d ** -0.5
            if causal:
                s = s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1), float("-inf"))
            want = s.softmax(-1) @ v[ks, h].double()
            # P and the result are rounded to 11 bits: 2^-11 max|v| each
            assert float((out[qs, h].double() - want).abs().max()) <= 2 ** -10 * float(v.abs().max())
