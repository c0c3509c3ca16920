"""Calls that something other than plain eager autograd watches: forward-mode tangents, traces, function
transforms and compiled autograd.  The functions refuse what the Python autograd classes refuse and give the
same numbers where those run."""
import pytest
import torch

from tests import _util as U

pytestmark = pytest.mark.gpu

LAYOUTS = ("qkv", "kv", "separate", "sparse")


def _call(layout, dropout_p=0.0, seed=0):
    """(function of the packed inputs, those inputs) of a small call."""
    from flash_attn_b200 import flash_attn_interface as fi
    from flash_attn_b200.flash_blocksparse_attn_interface import flash_blocksparse_attn_func
    lens = [150, 1, 77]
    q, k, v, _, cu, _ = U.make_varlen(lens, lens, 2, 64, torch.float16, seed=seed)
    s = max(lens)
    if layout == "qkv":
        return lambda x: fi.flash_attn_unpadded_qkvpacked_func(x, cu, s, dropout_p, causal=True), [torch.stack([q, k, v], 1)]
    if layout == "sparse":
        block = torch.ones(16, 1, dtype=torch.int32, device="cuda")
        return lambda x: flash_blocksparse_attn_func(x, cu, block, dropout_p, s), [torch.stack([q, k, v], 1)]
    if layout == "kv":
        return (lambda x, y: fi.flash_attn_unpadded_kvpacked_func(x, y, cu, cu, s, s, dropout_p),
                [q, torch.stack([k, v], 1)])
    return lambda x, y, z: fi.flash_attn_unpadded_func(x, y, z, cu, cu, s, s, dropout_p), [q, k, v]


@pytest.mark.parametrize("layout", LAYOUTS)
def test_forward_mode_tangents_are_refused(layout):
    import torch.autograd.forward_ad as fw
    f, x = _call(layout)
    with fw.dual_level():
        y = f(*x)   # no tangent: an ordinary call
        duals = [fw.make_dual(t, torch.ones_like(t)) if i == len(x) - 1 else t for i, t in enumerate(x)]
        with pytest.raises(NotImplementedError, match="jvp"):
            f(*duals)
    assert torch.equal(y, f(*x))


@pytest.mark.parametrize("layout", LAYOUTS)
def test_a_trace_replays_on_new_inputs(layout):
    f, x = _call(layout)
    traced = torch.jit.trace(lambda *a: f(*a) * 2, tuple(x), check_trace=False)
    new = _call(layout, seed=1)[1]
    poison = [torch.full((228, 2, 64), float("nan"), dtype=torch.float16, device="cuda") for _ in range(8)]
    del poison  # a replay that leaves its output unfilled finds these
    assert torch.equal(traced(*new), f(*new) * 2)


@pytest.mark.parametrize("layout", LAYOUTS)
def test_function_transforms_are_refused(layout):
    f, x = _call(layout)
    with pytest.raises(RuntimeError, match="setup_context"):
        torch.func.grad(lambda *a: f(*a).float().sum())(*x)
    with pytest.raises(RuntimeError, match="setup_context"):
        torch.vmap(lambda *a: f(*a))(*[t[None].expand(2, *t.shape) for t in x])


def _convert_cases():
    from flash_attn_b200.flash_blocksparse_attn_interface import convert_blockmask
    g = torch.Generator().manual_seed(3)
    a, b = [(torch.rand(64, 5, generator=g) < 0.4).int().cuda() for _ in range(2)]
    return convert_blockmask, a, b


def test_convert_blockmask_in_a_trace():
    convert, a, b = _convert_cases()
    traced = torch.jit.trace(lambda m: convert(m, False), (a,), check_trace=False)
    assert torch.equal(traced(b), convert(b, False))


def test_convert_blockmask_in_make_fx():
    from torch.fx.experimental.proxy_tensor import make_fx
    convert, a, b = _convert_cases()
    for mode in ("real", "fake"):
        graph = make_fx(lambda m: convert(m, True), tracing_mode=mode)(a)
        assert torch.equal(graph(b), convert(b, True)), mode


def test_convert_blockmask_under_vmap():
    convert, a, b = _convert_cases()
    got = torch.vmap(lambda m: convert(m, False))(torch.stack([a, b]))
    assert torch.equal(got, torch.stack([convert(a, False), convert(b, False)]))


def test_convert_blockmask_on_fake_tensors():
    from torch._subclasses.fake_tensor import FakeTensorMode
    convert, a, _ = _convert_cases()
    with FakeTensorMode() as mode:
        fake = convert(mode.from_tensor(a), False)
    assert fake.shape == (5, 64) and fake.dtype is torch.int32


def test_convert_blockmask_in_a_full_graph_compile():
    convert, a, b = _convert_cases()
    f = torch.compile(lambda m: convert(m, False), backend="eager", fullgraph=True)
    assert torch.equal(f(a), convert(a, False)) and torch.equal(f(b), convert(b, False))


def test_layouts_the_conversion_kernel_does_not_take():
    """Types whose zeros are not a bit pattern of their own, and empty layouts: what the framework operations
    accept and refuse."""
    convert, a, _ = _convert_cases()
    assert torch.equal(convert(a.to(torch.complex64), False), convert(a, False))
    assert convert(a[:0], False).shape == (5, 0)
    with pytest.raises(IndexError):
        convert(a[:, :0], False)


def test_unpad_input_in_a_trace():
    from flash_attn_b200 import bert_padding as bp
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(3, 40, 16, device="cuda", generator=g).half()
    mask = torch.arange(40, device="cuda")[None] < torch.tensor([[40], [7], [23]], device="cuda")
    traced = torch.jit.trace(lambda t, m: bp.unpad_input(t, m)[:3], (x, mask), check_trace=False)
    other = mask.flip(0, 1)   # as many valid tokens, elsewhere
    for got, want in zip(traced(x, other), bp.unpad_input(x, other)[:3]):
        assert torch.equal(got, want)


@pytest.mark.parametrize("compiler", ["graph", "dynamo"])
@pytest.mark.parametrize("layout,dropout_p", [("qkv", 0.0), ("qkv", 0.2), ("kv", 0.2), ("separate", 0.0), ("sparse", 0.1)])
def test_compiled_autograd_gives_the_same_gradients(layout, dropout_p, compiler):
    import torch._dynamo.compiled_autograd as ca
    from flash_attn_b200 import flash_attn_cuda as fc
    fc.options.deterministic = True
    try:
        for step in range(2):   # the second pass takes the graph of the first, with another mask
            grads = []
            for compiled in (False, True):
                f, x = _call(layout, dropout_p, seed=step)
                torch.cuda.manual_seed(5 + step)
                for t in x:
                    t.requires_grad_()
                out = f(*x)
                dout = torch.sin(torch.arange(out.numel(), device="cuda")).reshape(out.shape).half()
                if compiled:
                    with ca._enable((lambda gm: gm) if compiler == "graph" else lambda gm: torch.compile(gm, backend="eager")):
                        out.backward(dout)
                else:
                    out.backward(dout)
                grads.append([t.grad for t in x])
            for a, b in zip(*grads):
                assert torch.equal(a, b)
    finally:
        fc.options.deterministic = False
