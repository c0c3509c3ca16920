"""GPU tests of the mask index lists, the row copies and the rotary pass at the edges of their warps and
passes, against framework indexing (integers and copies: equal)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,seqlen", [(1, 1), (3, 255), (2, 256), (5, 257), (255, 3), (257, 40), (600, 33), (2, 5000)])
@pytest.mark.parametrize("density", [0.0, 0.5, 1.0])
def test_mask_lists_match_the_framework(batch, seqlen, density):
    from flash_attn_b200 import bert_padding as bp
    g = torch.Generator(device="cuda").manual_seed(batch + seqlen)
    mask = torch.rand(batch, seqlen, device="cuda", generator=g) < density
    assert bp._mask_kernel_path(mask)
    x = torch.randn(batch, seqlen, 8, device="cuda", generator=g).half()
    packed, idx, cu, longest = bp.unpad_input(x, mask)
    want_packed, want_idx, want_cu, want_longest = bp.unpad_input(x, mask.int())  # framework route
    assert idx.dtype is torch.int64 and cu.dtype is torch.int32 and isinstance(longest, int)
    assert torch.equal(idx, want_idx) and torch.equal(cu, want_cu) and longest == want_longest
    assert torch.equal(packed, want_packed)


def test_masks_that_keep_the_framework_route():
    from flash_attn_b200 import bert_padding as bp
    m = torch.ones(4, 6, dtype=torch.bool, device="cuda")
    assert not bp._mask_kernel_path(m.int()) and not bp._mask_kernel_path(m.t()) and not bp._mask_kernel_path(m.cpu())
    x = torch.randn(6, 4, 8, device="cuda").half()
    m[1, 2] = False
    packed, idx, _, _ = bp.unpad_input(x, m.t())
    assert torch.equal(packed, x.reshape(24, 8)[m.t().reshape(-1)]) and idx.numel() == 23


@pytest.mark.parametrize("units", [1, 2, 3, 31, 32, 33, 127, 128, 129, 288])
@pytest.mark.parametrize("rows", [1, 7, 257])
def test_row_copies(units, rows):
    from flash_attn_b200 import bert_padding as bp
    from flash_attn_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(units)
    x = torch.randn(rows + 5, units * 8, device="cuda", generator=g).half()
    idx = torch.randperm(rows + 5, device="cuda", generator=g)[:rows]
    got = bp.gather_rows(x, idx)
    assert torch.equal(got, x[idx])
    want = torch.zeros_like(x)
    want[idx] = got
    # whatever the workspace held before, also entries that look like row numbers
    for fill in (-1, 0, rows - 1, rows, 0x7fffffff):
        inverse = torch.full((rows + 5,), fill, dtype=torch.int32, device="cuda")
        out = torch.full_like(x, float("nan"))
        check(lib.fa_scatter_rows(got.data_ptr(), idx.data_ptr(), out.data_ptr(), rows, rows + 5, units * 16,
                                  inverse.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert torch.equal(out, want)


# head sizes that do and do not divide a warp, parts of one token below, at and above 128 units
@pytest.mark.parametrize("heads,d", [(1, 8), (5, 24), (16, 64), (17, 64), (8, 128), (9, 128), (32, 128), (3, 256)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_rotary_pass(heads, d, dtype):
    from flash_attn_b200.rotary import RotaryEmbedding
    rot = RotaryEmbedding(d).cuda()
    x = torch.randn(2, 19, 3, heads, d, device="cuda").to(dtype)
    assert rot.fused_path(x)
    got = rot.apply_qkv(x)
    q, k = rot(x[:, :, 0].double(), x[:, :, 1].double(), seq_dimension=-3)
    assert torch.equal(got[:, :, 2], x[:, :, 2])
    # one rounding to 16 bits of values up to |a| + |b|, fp32 angles on both sides
    ulp = 2.0 ** -11 if dtype is torch.float16 else 2.0 ** -8
    for i, want in enumerate((q, k)):
        bound = ulp * x[:, :, i].abs().max().item() * 2
        assert (got[:, :, i].double() - want).abs().max().item() <= bound


@pytest.mark.parametrize("batch,seqlen,kernels", [(16384, 2, True), (16385, 2, False), (2, 16384, True), (2, 16385, False)])
def test_masks_at_the_limit_of_the_list_kernels(batch, seqlen, kernels):
    """Longer sequences and larger batches, which the kernels are slow at, keep the framework route."""
    from flash_attn_b200 import bert_padding as bp
    mask = torch.rand(batch, seqlen, device="cuda") < 0.5
    assert bp._mask_kernel_path(mask) is kernels
    x = torch.randn(batch, seqlen, 8, device="cuda").half()
    for a, b in zip(bp.unpad_input(x, mask), bp.unpad_input(x, mask.int())):
        assert torch.equal(a, b) if torch.is_tensor(a) else a == b


@pytest.mark.parametrize("units", [1023, 1024, 1025, 2048, 5000])
@pytest.mark.parametrize("rows", [1, 9])
def test_long_rows_move_in_pieces(units, rows):
    from flash_attn_b200 import bert_padding as bp
    g = torch.Generator(device="cuda").manual_seed(units)
    x = torch.randn(rows + 3, units * 8, device="cuda", generator=g).half()
    idx = torch.randperm(rows + 3, device="cuda", generator=g)[:rows]
    got = bp.gather_rows(x, idx)
    assert torch.equal(got, x[idx])
    want = torch.zeros_like(x)
    want[idx] = got
    assert torch.equal(bp.scatter_rows(got, idx, rows + 3), want)
