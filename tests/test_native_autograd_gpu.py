"""The C++ autograd node behind the functional API and the Python autograd classes give the same outputs,
the same gradients and leave the generator in the same place."""
import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout,p,only_kv", [("qkv", 0.0, False), ("qkv", 0.2, False), ("kv", 0.2, True),
                                              ("separate", 0.1, False), ("sparse", 0.1, False)])
def test_native_node_matches_the_python_classes(layout, p, only_kv):
    from flash_attn_b200 import flash_attn_cuda as fc
    from flash_attn_b200 import flash_attn_interface as fi
    from flash_attn_b200.flash_blocksparse_attn_interface import flash_blocksparse_attn_func
    if fc.binding_in_use() != "compiled":
        pytest.skip("compiled binding not built")
    sq = [150, 1, 77]
    sk = sq if layout in ("qkv", "sparse") else [260, 40, 5]
    q, k, v, dout, cu_q, cu_k = U.make_varlen(sq, sk, 2, 64, torch.float16, seed=41)
    mq, mk = max(sq), max(sk)
    block = torch.ones(16, 1, dtype=torch.int32, device="cuda")

    def run():
        torch.cuda.manual_seed(17)
        if layout in ("qkv", "sparse"):
            x = [torch.stack([q, k, v], dim=1)]
        elif layout == "kv":
            x = [q.clone(), torch.stack([k, v], dim=1)]
        else:
            x = [q.clone(), k.clone(), v.clone()]
        for i, t in enumerate(x):
            t.requires_grad_(not (only_kv and i == 0))
        if layout == "qkv":
            out = fi.flash_attn_unpadded_qkvpacked_func(x[0], cu_q, mq, p, causal=True)
        elif layout == "sparse":
            out = flash_blocksparse_attn_func(x[0], cu_q, block, p, mq)
        elif layout == "kv":
            out = fi.flash_attn_unpadded_kvpacked_func(*x, cu_q, cu_k, mq, mk, p)
        else:
            out = fi.flash_attn_unpadded_func(*x, cu_q, cu_k, mq, mk, p, softmax_scale=0.2)
        between = torch.rand(1, device="cuda")  # the mask of the backward is the forward's all the same
        out.backward(dout)
        return out.detach(), [t.grad for t in x], between, torch.rand(1, device="cuda")

    fc.options.deterministic = True
    try:
        a = run()
        saved, fc._binding = fc._binding, None
        try:
            b = run()
        finally:
            fc._binding = saved
    finally:
        fc.options.deterministic = False
    assert torch.equal(a[0], b[0]) and torch.equal(a[2], b[2]) and torch.equal(a[3], b[3])
    for x, y in zip(a[1], b[1]):
        assert (x is None and y is None) or torch.equal(x, y)


def test_backward_twice_is_refused():
    from flash_attn_b200.flash_attn_interface import flash_attn_unpadded_qkvpacked_func
    q, k, v, dout, cu, _ = U.make_varlen([33], [33], 1, 64, torch.float16, seed=42)
    qkv = torch.stack([q, k, v], dim=1).requires_grad_()
    out = flash_attn_unpadded_qkvpacked_func(qkv, cu, 33, 0.0)
    out.backward(dout)
    with pytest.raises(RuntimeError, match="second time"):
        out.backward(dout)


def test_head_shard_changes_as_one_value():
    """Backward passes on the autograd thread while another thread enters and leaves head_shard: every pass sees one
    shard or the other, never the total of one with the offset of the other (which the call would refuse)."""
    import sys
    import threading
    from flash_attn_b200 import flash_attn_cuda as fc
    from flash_attn_b200.flash_attn_interface import flash_attn_unpadded_qkvpacked_func
    q, k, v, dout, cu, _ = U.make_varlen([16], [16], 2, 64, torch.float16, seed=1)
    qkv = torch.stack([q, k, v], dim=1).requires_grad_()
    stop = threading.Event()

    def toggle():
        while not stop.is_set():
            fc.options.mask_heads = (8, 6)
            fc.options.mask_heads = (2, 0)

    out = flash_attn_unpadded_qkvpacked_func(qkv, cu, 16, 0.1)
    thread = threading.Thread(target=toggle)
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)   # the two threads take turns on the interpreter
    thread.start()
    try:
        for _ in range(10000):
            torch.autograd.grad(out, qkv, dout, retain_graph=True)
    finally:
        stop.set()
        thread.join()
        sys.setswitchinterval(interval)
        fc.options.mask_heads = None


def _qkv(seed, n=50):
    q, k, v, dout, cu, _ = U.make_varlen([n], [n], 2, 64, torch.float16, seed=seed)
    return torch.stack([q, k, v], dim=1), dout, cu


def test_retained_graph_gives_the_same_gradient_twice():
    from flash_attn_b200.flash_attn_interface import flash_attn_unpadded_qkvpacked_func
    qkv, dout, cu = _qkv(43)
    qkv.requires_grad_()
    out = flash_attn_unpadded_qkvpacked_func(qkv, cu, 50, 0.2)
    a = torch.autograd.grad(out, qkv, dout, retain_graph=True)[0]
    b = torch.autograd.grad(out, qkv, dout)[0]
    assert torch.equal(a, b)   # one key tile: a single writer of dq


def test_a_saved_input_or_output_changed_in_place_is_refused():
    from flash_attn_b200.flash_attn_interface import flash_attn_unpadded_qkvpacked_func
    qkv, dout, cu = _qkv(44)
    leaf = qkv.clone().requires_grad_()
    x = leaf * 1
    out = flash_attn_unpadded_qkvpacked_func(x, cu, 50, 0.0)
    x.add_(1)
    with pytest.raises(RuntimeError, match="inplace"):
        out.backward(dout)
    out = flash_attn_unpadded_qkvpacked_func(leaf, cu, 50, 0.0)
    out.add_(1)
    with pytest.raises(RuntimeError, match="inplace"):
        out.backward(dout)


def test_saved_tensor_hooks_see_and_replace_what_is_saved():
    from flash_attn_b200.flash_attn_interface import flash_attn_unpadded_qkvpacked_func
    qkv, dout, cu = _qkv(45)
    grads = []
    for hooks in (False, True):
        x = qkv.clone().requires_grad_()
        torch.cuda.manual_seed(3)
        with torch.autograd.graph.save_on_cpu() if hooks else torch.enable_grad():
            out = flash_attn_unpadded_qkvpacked_func(x, cu, 50, 0.2)
        grads.append(torch.autograd.grad(out, x, dout)[0])
    assert torch.equal(*grads)


def test_packed_inputs_of_other_orders_and_strides():
    """Packed tensors that are not contiguous: heads before the three parts in memory, rows with a gap, an expanded
    gradient."""
    from flash_attn_b200.flash_attn_interface import flash_attn_unpadded_qkvpacked_func
    qkv, dout, cu = _qkv(46)
    want_x = qkv.clone().requires_grad_()
    want = flash_attn_unpadded_qkvpacked_func(want_x, cu, 50, 0.0, causal=True)
    want_g = torch.autograd.grad(want, want_x, dout[:1].expand_as(dout))[0]
    wide = torch.zeros(50, 4, 3, 64, dtype=torch.float16, device="cuda")
    wide[:, :3, :2] = qkv
    for x in (qkv.transpose(1, 2).contiguous().transpose(1, 2), wide[:, :3, :2]):
        x = x.detach().requires_grad_()
        assert not x.is_contiguous()
        out = flash_attn_unpadded_qkvpacked_func(x, cu, 50, 0.0, causal=True)
        assert torch.equal(out, want)
        assert torch.equal(torch.autograd.grad(out, x, dout[:1].expand_as(dout))[0], want_g)
