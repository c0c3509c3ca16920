"""GPU test of the backward for at most 256 queries at d = 64 with a causal mask, where two stages of K and V serve calls whose keys all
have queries: the same bits as calls of a few blocks, which hold one stage."""
import pytest
import torch

from tests import test_short_queries_gpu as short

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,dtype,p_dropout", [(32, torch.float16, 0.0), (64, torch.bfloat16, 0.0), (64, torch.float16, 0.2)])
@pytest.mark.parametrize("deterministic", [False, True])
def test_against_a_few_sequences_at_a_time(d, dtype, p_dropout, deterministic, monkeypatch):
    monkeypatch.setattr(short, "LENS_K", [128, 40, 129, 256, 0, 250, 100, 200, 1, 130] * 4)
    short.test_against_a_few_sequences_at_a_time(d, dtype, p_dropout, True, deterministic)
