"""The native calls on the packed projection (norm + attention in one autograd node; norm + cache append in one
launch) against the general path of the same module, and the vectorised norm kernels at the edges of their warps."""
import ctypes as C
from functools import partial

import pytest
import torch

from simplicial_attention_b200 import SlidingWindowTwoSimplicialMHA, _lib, sliding_two_simplicial_attn
from simplicial_attention_b200.headnorm import head_rmsnorm

pytestmark = pytest.mark.gpu


@pytest.fixture
def native(monkeypatch):
    """Names of the native module calls that answered (a None sends the module to its general path)."""
    real, answered = _lib.ext(), []

    class Counted:
        def __getattr__(self, name):
            f = getattr(real, name)
            if name not in ("qkv_attn", "qkv_attn_cached", "step"):
                return f

            def call(*args):
                res = f(*args)
                if res is not None:
                    answered.append(name)
                return res
            return call

    monkeypatch.setattr(_lib, "ext", lambda: Counted())
    return answered


def _module(hq, hk, d, w1, w2, dtype, seed=0):
    torch.manual_seed(seed)
    m = SlidingWindowTwoSimplicialMHA(dim=64, dim_head=d, heads=hq, key_value_heads=hk, prenorm=True, w1=w1, w2=w2).to("cuda", dtype)
    with torch.no_grad():
        for p in m.parameters():
            if p.dim() == 1:
                p.add_(0.1 * torch.randn_like(p))
    return m


def _general(m):
    """The same module with an attend the native calls do not recognise."""
    at = m.attend
    m.attend = lambda q, k, v: at(q, k, v)
    return m


@pytest.mark.parametrize("hq,hk,d,n,dtype,autocast", [
    (4, 4, 64, 70, torch.float32, False),
    (6, 2, 32, 33, torch.float32, False),      # 14 heads of 32: the last warp of a row is part empty
    (3, 1, 128, 40, torch.bfloat16, False),
    (8, 4, 64, 130, torch.float32, True),
])
def test_training_pass_equals_the_general_path(native, hq, hk, d, n, dtype, autocast):
    res = []
    for general in (False, True):
        m = _module(hq, hk, d, 24, 5, dtype)
        if general:
            _general(m)
        x = torch.randn(2, n, 64, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).to(dtype).requires_grad_()
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=autocast):
            out = m(x)
        assert native == ["qkv_attn"]           # the first module's call, and none of the second's
        out.backward(torch.randn(out.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(2)).to(out.dtype))
        res.append([out.detach(), x.grad] + [p.grad for p in m.parameters()])
    tol = 1e-5 if dtype == torch.float32 and not autocast else 1e-2
    for a, b in zip(*res):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert (a - b).float().norm() <= tol * b.float().norm()


@pytest.mark.parametrize("b,hq,hk,d,dtype,prompt", [
    (1, 2, 2, 64, torch.bfloat16, 3),          # windows not yet full
    (3, 4, 2, 32, torch.bfloat16, 40),
    (2, 2, 1, 128, torch.float32, 17),
])
def test_generation_equals_the_general_path(native, b, hq, hk, d, dtype, prompt):
    w1, w2 = 20, 4
    fast, slow = _module(hq, hk, d, w1, w2, dtype), _general(_module(hq, hk, d, w1, w2, dtype))
    x = torch.randn(b, prompt + 6, 64, device="cuda").to(dtype)
    with torch.no_grad():
        states = [m(x[:, :prompt], return_cache=True)[1] for m in (fast, slow)]
        at = prompt
        for new in (1, 1, 3, 1):
            got = [m(x[:, at:at + new], cache=c, return_cache=True) for m, c in zip((fast, slow), states)]
            at += new
            states = [g[1] for g in got]
            assert (got[0][0] - got[1][0]).float().norm() <= 1e-2 * got[1][0].float().norm()
            for s, t in zip(*states):
                for a, c in zip(s, t):
                    assert a.shape == c.shape and (a - c).float().norm() <= 1e-2 * c.float().norm()
    assert native == ["step"] * 4


@pytest.mark.parametrize("dim,pre,post,hook", [
    (512, True, True, False),                  # the widest row of the norm kernel
    (96, True, False, False),                  # a width it does not take
    (64, False, False, False),
    (64, True, False, True),                   # a hooked submodule has to be called
])
def test_generation_step_of_plain_and_hooked_modules(native, dim, pre, post, hook):
    torch.manual_seed(0)
    m = SlidingWindowTwoSimplicialMHA(dim=dim, dim_head=64, heads=4, key_value_heads=2, prenorm=pre, postnorm=post, w1=20, w2=4)
    m = m.to("cuda", torch.bfloat16)
    calls = []
    if hook:
        m.to_qkv.register_forward_hook(lambda *a: calls.append(1))
    x = torch.randn(2, 30, dim, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        want = m(x)
        _, cache = m(x[:, :25], return_cache=True)
        calls.clear()
        native.clear()
        got, _ = m(x[:, 25:], cache=cache, return_cache=True)
    assert bool(calls) == hook and native == ["qkv_attn_cached" if hook else "step"]
    assert (got - want[:, 25:]).float().norm() <= 1e-2 * want[:, 25:].float().norm()


@pytest.mark.parametrize("rows,k,outs", [(1, 32, 16), (8, 64, 48), (9, 288, 64), (15, 512, 1536), (16, 2080, 128)])
def test_projection_of_few_rows(rows, k, outs):
    g = torch.Generator("cuda").manual_seed(rows)
    x, w = (torch.randn(s, k, device="cuda", generator=g).to(torch.bfloat16) for s in (rows, outs))
    y = torch.full((rows + 1, outs), 7., device="cuda", dtype=torch.bfloat16)
    _lib.check(_lib.lib().sa2_rows_linear(*(C.c_void_p(t.data_ptr()) for t in (x, w, y)), rows, k, outs,
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream)), "sa2_rows_linear")
    want = x.float() @ w.float().t()
    assert (y[:rows].float() - want).abs().max() <= 1e-2 * want.abs().max()
    assert (y[rows] == 7).all()


def test_other_attend_callables_still_run(native):
    m = _module(2, 2, 64, 16, 4, torch.float32)
    x = torch.randn(1, 30, 64, device="cuda")
    ref = m(x)
    m.attend = partial(sliding_two_simplicial_attn, w1=16, w2=4, kernel="simt")
    assert torch.allclose(m(x), ref, atol=1e-5)
    assert native == ["qkv_attn"] * 2
    m.attend = lambda q, k, v: sliding_two_simplicial_attn(q, k, v, w1=16, w2=4)
    assert torch.allclose(m(x), ref, atol=1e-5) and native == ["qkv_attn"] * 2
    with pytest.raises(KeyError):
        m.attend = partial(sliding_two_simplicial_attn, w1=16, w2=4, kernel="other")
        m(x)


@pytest.mark.parametrize("rows,channels,d,offset", [(1, 32, 32, 0), (7, 96, 32, 0), (1000, 1536, 512, 0), (65, 6400, 64, 0), (5, 128, 64, 1)])
def test_norm_edges(rows, channels, d, offset):
    """Part-empty warps, a whole row per warp, the widest projection of the backward, rows off 16-byte boundaries."""
    base = torch.randn(rows, channels + offset, device="cuda")
    x = base[:, offset:].detach().requires_grad_()
    gain = (1 + 0.1 * torch.randn(channels, device="cuda")).requires_grad_()
    dy = torch.randn(rows, channels, device="cuda")
    y = head_rmsnorm(x, gain, d, 1e-6)
    y.backward(dy)
    xd, gd = x.detach().double().requires_grad_(), gain.detach().double().requires_grad_()
    xh = xd.view(rows, -1, d) if offset == 0 else xd.reshape(rows, -1, d)
    ref = (xh * torch.rsqrt(xh.pow(2).mean(-1, keepdim=True) + 1e-6)).reshape(rows, -1) * gd
    ref.backward(dy.double())
    for a, c in ((y, ref), (x.grad, xd.grad), (gain.grad, gd.grad)):
        assert (a.double() - c).norm() <= 1e-5 * c.norm()
