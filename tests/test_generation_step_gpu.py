"""The one-token kernel of generation (norms, cache hand-over and attention in one launch) and the projections of up to 64 rows:
remainders of keys, offsets and heads, and short caches against the same module called module by module; over-long and strided caches,
and the shapes that the kernel takes or leaves, at its C entry against 64 bits; second values that are not finite."""
import ctypes as C

import pytest
import torch

import simplicial_attention_b200 as sa
from simplicial_attention_b200 import _lib

pytestmark = pytest.mark.gpu
# Results are bf16 (2^-9 each) behind two projections of bf16 operands whose rounded inputs may differ by one unit in the last place
# (2^-8) in either path; measured 1e-3 to 1e-2.
REL = 2e-2

CASES = [
    # b, hq, hk, d, w1, w2, prompt, prenorm, postnorm
    (1, 8, 4, 64, 512, 32, 512, True, False),        # eight CTAs a head
    (3, 8, 4, 64, 512, 32, 5, True, False),          # caches shorter than the windows
    (2, 4, 4, 128, 700, 40, 800, True, False),
    (5, 8, 1, 64, 100, 64, 130, True, False),        # 32 blocks of rows for eight warps
    (2, 3, 1, 64, 64, 8, 70, False, False),
    (2, 1, 1, 64, 1, 1, 9, True, False),             # nothing to keep
    (64, 2, 1, 128, 77, 17, 200, True, False),
    (7, 8, 4, 64, 2000, 32, 2100, True, False),      # several pieces of a stretch
    (33, 8, 4, 64, 512, 32, 512, True, True),        # projections of more than 32 rows
    (2, 4, 2, 64, 100, 65, 130, True, False),        # a second window that the kernel does not take
    (2, 4, 2, 32, 100, 8, 130, True, False),         # nor this head dim
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%d_hq%d_hk%d_d%d_w%d_%d_n%d_%d%d" % c)
def test_step_matches_the_modules(case):
    b, hq, hk, d, w1, w2, n, pre, post = case
    torch.manual_seed(n)
    m = sa.SlidingWindowTwoSimplicialMHA(dim=hq * d, dim_head=d, heads=hq, key_value_heads=hk, prenorm=pre, postnorm=post, w1=w1, w2=w2)
    m = m.to("cuda", torch.bfloat16)
    with torch.no_grad():
        for norm in (m.q_norm, *m.k_norms, *m.v_norms):
            norm.weight.uniform_(0.5, 1.5)
        _, cache = m(torch.randn(b, n, hq * d, device="cuda", dtype=torch.bfloat16), return_cache=True)
        for _ in range(2):                            # the second step on the caches that the first one made
            x = torch.randn(b, 1, hq * d, device="cuda", dtype=torch.bfloat16)
            out, new = m(x, cache=cache, return_cache=True)
            hook = m.to_qkv.register_forward_hook(lambda *a: None)       # a hook is seen by the modules only
            want, want_new = m(x, cache=cache, return_cache=True)
            hook.remove()
            assert sa.device_status() == 0 and out.shape == want.shape
            assert (out.float() - want.float()).norm() <= REL * want.float().norm()
            for got, ref in zip((t for s in new for t in s), (t for s in want_new for t in s)):
                assert got.shape == ref.shape
                # (one unit in the last place where the projections' sums round to either side)
                assert ((got.float() - ref.float()).abs() <= 2 ** -6 * ref.float().abs() + 1e-3).all()
            cache = new


def test_nan_key_reaches_its_head_only():
    """A NaN in one head's cached keys makes that head's outputs NaN, and the other sequences' none."""
    torch.manual_seed(0)
    m = sa.SlidingWindowTwoSimplicialMHA(dim=256, dim_head=64, heads=4, key_value_heads=2, prenorm=True, w1=64, w2=8).to("cuda", torch.bfloat16)
    with torch.no_grad():
        _, cache = m(torch.randn(2, 80, 256, device="cuda", dtype=torch.bfloat16), return_cache=True)
        cache[0][0][1, 30, 0, 5] = float("nan")
        out, _ = m(torch.randn(2, 1, 256, device="cuda", dtype=torch.bfloat16), cache=cache, return_cache=True)
    assert out[0].isfinite().all() and out[1].isnan().all()


class _NormArgs(C.Structure):
    _fields_ = [("x", C.c_void_p), ("dy", C.c_void_p), ("y", C.c_void_p), ("rstd", C.c_void_p), ("gain", C.c_void_p * 5), ("dgain", C.c_void_p * 5),
                ("partial", C.c_void_p), ("partial_bytes", C.c_size_t), ("rows", C.c_int64), ("x_stride", C.c_int64), ("y_stride", C.c_int64),
                ("dy_stride", C.c_int64), ("hq", C.c_int32), ("hk", C.c_int32), ("d", C.c_int32), ("x_dtype", C.c_int32), ("y_dtype", C.c_int32),
                ("gain_dtype", C.c_int32), ("eps", C.c_float), ("stream", C.c_void_p)]


class _Set(C.Structure):
    _fields_ = [("cache", C.c_void_p), ("strides", _lib.Strides), ("dst", C.c_void_p), ("keep", C.c_int32)]


def _step_attn(proj, gains, caches, hq, hk, d, w1, w2):
    """(status, out, new caches) of sa2_step_attn; caches [k, k', v, v'], each [b][keep][hk][d]."""
    b = proj.shape[0]
    a = _NormArgs(x=proj.data_ptr(), rows=b, x_stride=proj.stride(0), hq=hq, hk=hk, d=d, x_dtype=_lib.SA2_BF16, y_dtype=_lib.SA2_BF16,
                  gain_dtype=_lib.SA2_BF16, eps=1e-6, stream=torch.cuda.current_stream().cuda_stream)
    for v in range(5):
        a.gain[v] = gains[v].data_ptr()
    sets, new = (_Set * 4)(), []
    for s, c in enumerate(caches):
        keep = c.shape[1]
        new.append(torch.empty(b, min(keep + 1, (w2 if s & 1 else w1) - 1), hk, d, device="cuda", dtype=torch.bfloat16))
        sets[s] = _Set(c.data_ptr(), _lib.Strides(*c.stride()[:3]), new[s].data_ptr(), keep)
    out = torch.empty(b, hq, d, device="cuda", dtype=torch.bfloat16)
    fn = _lib.lib().sa2_step_attn
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32, C.c_int32, C.c_int32, C.c_float]
    return fn(C.byref(a), sets, out.data_ptr(), b, w1, w2, d ** -0.5), out, new


def _step_inputs(b, hq, hk, d, keep1, keep2):
    g = torch.Generator(device="cuda").manual_seed(hq + keep1)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    proj, gains = rand(b, d * (hq + 4 * hk)), [(1 + 0.2 * rand(d)).to(torch.bfloat16) for _ in range(5)]
    # every cache a window of a wider tensor: other rows, heads and channels around it
    caches = [rand(b, keep + 3, 2 * hk, d + 8)[:, 2:2 + keep, 1:1 + hk, 8:] for keep in (keep1, keep2, keep1, keep2)]
    return proj, gains, caches


def _step_reference(proj, gains, caches, hq, hk, d, w1, w2):
    """Rows as the kernel rounds them, then 64 bits: (out, the five kinds of new rows)."""
    b = proj.shape[0]
    x = proj.float().view(b, hq + 4 * hk, d)
    x = x * (x.square().mean(-1, keepdim=True) + 1e-6).rsqrt()
    kv = x[:, hq:].view(b, 2, hk, 2, d)
    rows = [x[:, :hq], kv[:, 0, :, 0], kv[:, 0, :, 1], kv[:, 1, :, 0], kv[:, 1, :, 1]]
    q, *new = [(r * g.float()).to(torch.bfloat16) for r, g in zip(rows, gains)]
    k1, k2, v1, v2 = [torch.cat((c, n[:, None]), 1)[:, -w:].double().repeat_interleave(hq // hk, 2)
                      for c, n, w in zip(caches, new, (w1, w2, w1, w2))]
    s = torch.einsum("bhc,bjhc,bkhc->bhjk", q.double(), k1, k2) * d ** -0.5
    p = s.flatten(-2).softmax(-1).view_as(s)
    return torch.einsum("bhjk,bjhc,bkhc->bhc", p, v1, v2), new


ENTRY = [
    # b, hq, hk, d, w1, w2, keep1, keep2
    (2, 4, 2, 64, 64, 8, 90, 30),           # caches longer than the windows
    (1, 8, 1, 64, 300, 17, 411, 16),
    (3, 2, 2, 128, 70, 64, 69, 100),
    (2, 3, 3, 64, 40, 33, 12, 40),          # the first one shorter, the second one longer
    (1, 1, 1, 64, 1, 1, 5, 5),
    (2, 2, 1, 128, 513, 32, 600, 3),
]


@pytest.mark.parametrize("case", ENTRY, ids=lambda c: "b%d_hq%d_hk%d_d%d_w%d_%d_keep%d_%d" % c)
def test_entry_takes_long_and_strided_caches(case):
    b, hq, hk, d, w1, w2, keep1, keep2 = case
    proj, gains, caches = _step_inputs(b, hq, hk, d, keep1, keep2)
    status, out, new = _step_attn(proj, gains, caches, hq, hk, d, w1, w2)
    assert status == _lib.SA2_OK
    want, rows = _step_reference(proj, gains, caches, hq, hk, d, w1, w2)
    # only operands and result are rounded; a row's norm may differ by one unit in its last place (2^-8) in a few entries
    assert (out.double() - want).norm() <= 2 ** -7 * want.norm()
    for n, c, r, w in zip(new, caches, rows, (w1, w2, w1, w2)):
        whole = torch.cat((c, r[:, None]), 1)[:, max(0, c.shape[1] + 2 - w):]
        assert n.shape == whole.shape
        if n.shape[1]:
            assert torch.equal(n[:, :-1], whole[:, :-1])
            assert ((n[:, -1].float() - whole[:, -1].float()).abs() <= 2 ** -7 * whole[:, -1].float().abs()).all()


def test_entry_leaves_what_it_does_not_take():
    for d, w2 in ((64, 65), (32, 8)):
        proj, gains, caches = _step_inputs(1, 2, 1, d, 20, 20)
        assert _step_attn(proj, gains, caches, 2, 1, d, 30, w2)[0] == 2        # SA2_ERR_UNSUPPORTED


@pytest.mark.parametrize("d,w1,w2", [(64, 100, 9), (128, 100, 16), (64, 700, 33)])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), 3e38, float("nan")])
@pytest.mark.parametrize("row", [0, 3, -1])
def test_second_values_that_are_not_finite(d, w1, w2, value, row):
    """Infinite second values reach the outputs of their channel as infinities of the sign that the sum over all keys has."""
    b, hq, hk = 2, 4, 2
    proj, gains, caches = _step_inputs(b, hq, hk, d, w1 + 20, w2 - 1)
    caches[3][1, row, 0, 5] = value
    status, out, _ = _step_attn(proj, gains, caches, hq, hk, d, w1, w2)
    want = _step_reference(proj, gains, caches, hq, hk, d, w1, w2)[0].to(torch.bfloat16)
    assert status == _lib.SA2_OK
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf()) and torch.equal(out[out.isinf()], want[want.isinf()])
    rest = want.isfinite() & (want.abs() < 1e30)
    assert (out[rest].double() - want[rest].double()).norm() <= 2 ** -7 * want[rest].double().norm()
    big = want.isfinite() & ~rest
    assert ((out[big].double() - want[big].double()).abs() <= 2 ** -4 * want[big].double().abs()).all()
