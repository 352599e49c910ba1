"""The native host path takes plain tensors of one device; anything else goes to the general path, which raises torch's
own errors or dispatches to the tensor's class.  Fake tensors stand for tensors of several GPUs and of a subclass, so
this runs without one."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

import simplicial_attention_b200 as sa
from simplicial_attention_b200 import _lib

B, DIM, HQ, HK, D, W1, W2 = 2, 128, 2, 1, 64, 16, 8
CHANNELS = D * (HQ + 4 * HK)


def _fake(on_second=()):
    """Arguments of a generation step; the tensors named in ``on_second`` sit on another GPU than the rest."""
    shapes = {"x": (B, 1, DIM), "proj": (B, 1, CHANNELS), "pre": (DIM,), "w_qkv": (CHANNELS, DIM), "gain": (D,), "w_out": (DIM, HQ * D), "post": (DIM,),
              "c1": (B, W1 - 1, HK, D), "c2": (B, W2 - 1, HK, D)}
    with FakeTensorMode():
        t = {k: torch.empty(s, dtype=torch.bfloat16, device=f"cuda:{int(k in on_second)}") for k, s in shapes.items()}
    return t, [t["gain"]] * 5, [t["c1"], t["c2"], t["c1"], t["c2"]]


@pytest.mark.parametrize("on_second", [(), ("w_qkv",), ("w_out",), ("gain",), ("c1",), ("pre",), ("post",)], ids=lambda s: "+".join(s) or "none")
def test_generation_calls_decline(on_second):
    t, gains, cache = _fake(on_second)
    ext = _lib.ext()
    assert ext.step(t["x"], t["pre"], 1e-6, t["w_qkv"], gains, cache, HQ, HK, D, 1e-6, W1, W2, 0, t["w_out"], t["post"], 1e-6) is None
    assert ext.qkv_attn_cached(t["proj"], gains, cache, HQ, HK, D, 1e-6, W1, W2, 0) is None
    assert ext.qkv_attn(t["proj"], gains, HQ, HK, D, 1e-6, torch.bfloat16, W1, W2, 0) is None


class Wrapped(torch.Tensor):
    """A weight whose values are elsewhere, as quantised weights are."""

    @staticmethod
    def __new__(cls, inner):
        return torch.Tensor._make_wrapper_subclass(cls, inner.shape, dtype=inner.dtype, device=inner.device)

    def __init__(self, inner):
        self.inner = inner

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        un = lambda a: a.inner if isinstance(a, Wrapped) else a
        res = func(*torch.utils._pytree.tree_map(un, args), **torch.utils._pytree.tree_map(un, kwargs or {}))
        return cls(res) if func is torch.ops.aten.detach.default else res


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["to_qkv", "combine_heads", "q_norm"])
def test_subclass_weights_are_dispatched(name):
    torch.manual_seed(0)
    m = sa.SlidingWindowTwoSimplicialMHA(dim=DIM, dim_head=D, heads=HQ, key_value_heads=HK, prenorm=True, w1=W1, w2=W2).cuda().bfloat16()
    x = torch.randn(B, 20, DIM, device="cuda").bfloat16()
    with torch.no_grad():
        _, cache = m(x, return_cache=True)
        want = m(x[:, :1], cache=cache, return_cache=True)[0]
        layer = getattr(m, name)
        layer.weight = torch.nn.Parameter(Wrapped(layer.weight.detach()), requires_grad=False)
        got = m(x[:, :1], cache=cache, return_cache=True)[0]
    assert (got.float() - want.float()).abs().max().item() <= 2e-2      # roundings of bf16 results of about 1


def _module():
    torch.manual_seed(0)
    m = sa.SlidingWindowTwoSimplicialMHA(dim=DIM, dim_head=D, heads=HQ, key_value_heads=HK, prenorm=True, postnorm=True, w1=W1, w2=W2)
    return m.cuda().bfloat16().requires_grad_(False), torch.randn(B, 20, DIM, device="cuda").bfloat16()


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["op", "module", "generation"])
def test_traced_calls_compute(what):
    """A trace replayed on other inputs gives their results (a trace of raw launches would return fresh, unwritten memory)."""
    m, x = _module()
    _, cache = m(x, return_cache=True)
    if what == "op":
        f = lambda q, k1, k2, v1, v2: sa.sliding_two_simplicial_attn(q, (k1, k2), (v1, v2), w1=W1, w2=W2)
        first, other = ([torch.randn(1, 50, h, D, device="cuda").bfloat16() for h in (HQ, HK, HK, HK, HK)] for _ in range(2))
    elif what == "module":
        f, first, other = m, [x], [x.flip(1).contiguous()]
    else:
        f = lambda t, a, b, c, d: m(t, cache=((a, b), (c, d)), return_cache=True)[0]
        first, other = ([x[:, i:i + 1].contiguous(), *cache[0], *cache[1]] for i in (0, 7))
    with torch.no_grad():
        traced = torch.jit.trace(f, tuple(first), check_trace=False)
        got, want = traced(*other), f(*other)
    assert (got.float() - want.float()).abs().max().item() <= 2 ** -5      # two roundings to bf16 of values below 4


@pytest.mark.gpu
def test_tangents_and_transforms_are_refused_not_dropped():
    import torch.autograd.forward_ad as fa
    m, x = _module()
    _, cache = m(x, return_cache=True)
    q, k1, k2, v1, v2 = (torch.randn(1, 50, h, D, device="cuda") for h in (HQ, HK, HK, HK, HK))
    op = lambda t: sa.sliding_two_simplicial_attn(t, (k1, k2), (v1, v2), w1=W1, w2=W2)
    with torch.no_grad(), fa.dual_level():
        with pytest.raises(NotImplementedError):
            m(fa.make_dual(x[:, :1].contiguous(), x[:, 1:2].contiguous()), cache=cache, return_cache=True)
        with pytest.raises(NotImplementedError):
            op(fa.make_dual(q, q))
    with pytest.raises(RuntimeError):
        torch.vmap(op)(q[None])
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: op(t).sum())(q)


@pytest.mark.gpu
def test_undefined_output_gradient_gives_zeros():
    """A consumer that returns no gradient leaves zeros on the operands, not None."""
    class Drop(torch.autograd.Function):
        @staticmethod
        def forward(ctx, t):
            return t.sum()

        @staticmethod
        def backward(ctx, g):
            return None

    ins = [torch.randn(1, 50, h, D, device="cuda").requires_grad_() for h in (HQ, HK, HK, HK, HK)]
    Drop.apply(sa.sliding_two_simplicial_attn(ins[0], ins[1:3], ins[3:5], w1=W1, w2=W2)).backward()
    assert all(t.grad is not None and not t.grad.any() for t in ins)


@pytest.mark.gpu
@pytest.mark.parametrize("limit,modules_run", [(CHANNELS, False), (CHANNELS - 1, True)])
def test_lowered_channel_limit_runs_the_norm_modules(limit, modules_run):
    m, x = _module()
    m.fused_head_norm_max_channels = limit
    calls = []
    m.q_norm.register_forward_hook(lambda *a: calls.append(1))
    m(x)
    assert bool(calls) == modules_run


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_python_function_equals_the_native_node(dtype):
    """The autograd function behind the calls that the native node declines: same bits, forward and backward."""
    cls = sa.SlidingTwoSimplicialAttention
    ins = [torch.randn(2, 70, h, D, device="cuda").to(dtype).requires_grad_() for h in (HQ, HK, HK, HK, HK)]
    dout = torch.randn(2, 70, HQ, D, device="cuda").to(dtype)
    res = []
    for apply in (cls.apply, super(cls, cls).apply):
        out, lse = apply(*ins, W1, W2, True, None, "auto", True)
        assert not lse.requires_grad
        res.append([out, lse, *torch.autograd.grad(out, ins, dout)])
    assert all(torch.equal(a, b) for a, b in zip(*res))
