"""The layout conversion and block-visit table kernels: list lengths around the 32-entry and 256-row steps they work
in, every element type, strided layouts, and the zero rows outside the sequences."""
import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("rows,cols,density", [(1, 1, 1.0), (16, 1, 0.5), (31, 3, 0.5), (256, 16, 0.25), (257, 17, 0.9),
                                               (1024, 64, 0.05), (520, 33, 0.0)])
def test_convert_blockmask_matches_the_framework_version(rows, cols, density, causal):
    from flash_attn_b200.flash_blocksparse_attn_interface import convert_blockmask
    torch.manual_seed(rows + cols)
    layout = (torch.rand(rows, cols) < density).to(torch.int32)
    want = convert_blockmask(layout, causal)   # CPU: framework operations
    for dt in (torch.bool, torch.int32, torch.int64, torch.float32, torch.float16, torch.uint8):
        assert torch.equal(convert_blockmask(layout.to(dt).cuda(), causal).cpu(), want), dt
    wide = torch.full((rows, 2 * cols), -0.0, device="cuda")
    wide[:, ::2] = layout.cuda().float() * -3.0
    assert torch.equal(convert_blockmask(wide[:, ::2], causal).cpu(), want)


@pytest.mark.parametrize("lens", [[1, 256, 257], [500, 31], [1000]])
def test_rows_outside_the_sequences_are_zero(lens):
    """A token buffer with rows in front of the first and behind the last sequence."""
    from flash_attn_b200 import flash_attn_cuda as fc
    from flash_attn_b200.flash_blocksparse_attn_interface import convert_blockmask
    s = max(lens)
    kb = (s + 255) // 256
    torch.manual_seed(1)
    layout = ((torch.rand(kb, kb) < 0.5) | torch.eye(kb, dtype=torch.bool)).repeat_interleave(16, dim=0).cuda()
    conv = convert_blockmask(layout, False)
    q, k, v, _, cu, _ = U.make_varlen(lens, lens, 2, 64, torch.float16, seed=5)
    pad = [torch.cat([torch.full_like(t[:1], 3.0).expand(7, -1, -1), t, t[:1].expand(9, -1, -1)]) for t in (q, k, v)]
    garbage = torch.full((1 << 20,), float("nan"), device="cuda", dtype=torch.float16)  # what the allocator hands out next
    del garbage
    out = fc.fwd_block(*pad, cu + 7, cu + 7, conv, s, s, 0.0, 0.125, False, False, None)[0]
    want = fc.fwd_block(q, k, v, cu, cu, conv, s, s, 0.0, 0.125, False, False, None)[0]
    assert torch.equal(out[7:7 + sum(lens)], want)
    assert not out[:7].any() and not out[7 + sum(lens):].any()


def _poisoned(shape, call):
    """call()[0] in memory that held NaN: every free block of its size is filled first."""
    garbage = [torch.full(shape, float("nan"), device="cuda", dtype=torch.float16) for _ in range(64)]
    nbytes = garbage[0].numel() * 2
    ranges = [(g.data_ptr(), g.data_ptr() + nbytes) for g in garbage]
    del garbage
    out = call()[0]
    assert any(lo <= out.data_ptr() < hi for lo, hi in ranges), "the allocator handed out other memory"
    return out


@pytest.mark.parametrize("front,behind", [(0, 0), (1, 0), (0, 1), (2999, 4001), (20000, 3)])
def test_unused_rows_of_a_token_buffer_are_zero(front, behind):
    from flash_attn_b200 import flash_attn_cuda as fc
    lens = [300, 0, 77]
    n = sum(lens)
    conv = torch.full((2, 32), -1, dtype=torch.int32, device="cuda")
    conv[:, :19] = 4 * torch.arange(19, device="cuda")   # every block of the longest sequence
    q, k, v, _, cu, _ = U.make_varlen(lens, lens, 2, 64, torch.float16, seed=6)
    pad = [torch.nn.functional.pad(t, (0, 0, 0, 0, front, behind), value=3.0) for t in (q, k, v)]
    out = _poisoned(pad[0].shape, lambda: fc.fwd_block(*pad, cu + front, cu + front, conv, 300, 300, 0.0, 0.125, False, False, None))
    want = fc.fwd_block(q, k, v, cu, cu, conv, 300, 300, 0.0, 0.125, False, False, None)[0]
    assert torch.equal(out[front:front + n], want) and want.any()
    assert not out[:front].any() and not out[front + n:].any()


def test_rows_beyond_the_covered_tiles_are_zero():
    """A sequence longer than the 128 rows max_seqlen_q announces."""
    from flash_attn_b200 import flash_attn_cuda as fc
    q, k, v, _, cu_q, cu_k = U.make_varlen([300, 13], [128, 13], 2, 64, torch.float16, seed=7)
    conv = (4 * torch.arange(16, dtype=torch.int32, device="cuda"))[None].contiguous()
    out = _poisoned(q.shape, lambda: fc.fwd_block(q, k, v, cu_q, cu_k, conv, 128, 128, 0.0, 0.125, False, False, None))
    assert not out[128:300].any()
    assert torch.isfinite(out).all() and out[:128].any() and out[300:].any()


@pytest.mark.parametrize("zero_unused,strided", [(0, False), (1, False), (1, True)])
def test_c_entry_points_and_rows_outside_the_sequences(zero_unused, strided):
    """fa_fwd writes the rows of the sequences and no others; fa_fwd_ex zeroes the others on request, unless o has a
    row stride of its own."""
    import ctypes
    from flash_attn_b200 import flash_attn_cuda as fc
    from flash_attn_b200._lib import check, lib
    lens, front, behind, heads, d = [200, 57], 5, 9, 2, 64
    n = sum(lens)
    conv = (4 * torch.arange(16, dtype=torch.int32, device="cuda"))[None].contiguous()
    q, k, v, _, cu, _ = U.make_varlen(lens, lens, heads, d, torch.float16, seed=8)
    want = fc.fwd_block(q, k, v, cu, cu, conv, 200, 200, 0.0, 0.125, False, False, None)[0]
    pad = [torch.nn.functional.pad(t, (0, 0, 0, 0, front, behind), value=3.0) for t in (q, k, v)]
    total = n + front + behind
    wide = torch.full((total, heads + (1 if strided else 0), d), 7.0, dtype=torch.float16, device="cuda")
    o = wide[:, :heads]
    lse = torch.empty(2, heads, 208, device="cuda")
    shifted = cu + front
    p = fc._make_fwd((2, total, total, heads, d), *pad, o, lse, shifted, shifted, 200, 200, 0.0, 0.125, False, 0, 0)
    ws = fc._bs_workspace(q.device, 2, conv)
    p.blockmask, (p.blockmask_rows, p.blockmask_cols) = conv.data_ptr(), conv.shape
    p.bs_workspace, p.bs_workspace_bytes = ws.data_ptr(), ws.numel()
    if zero_unused:
        check(lib.fa_fwd_ex(ctypes.byref(p), 1, fc._raw_stream()))
    else:
        check(lib.fa_fwd(ctypes.byref(p), fc._raw_stream()))
    assert torch.equal(o[front:front + n], want)
    outside = torch.cat([wide[:front], wide[front + n:]])
    assert (outside == (0.0 if zero_unused and not strided else 7.0)).all()
    if strided:
        assert (wide[:, heads] == 7.0).all()
