"""Keys and values that repeat a dimension (expanded tensors: one key/value set for a batch, or for all heads, or one row
for the whole sequence), which TMA cannot load in place."""
import ctypes as C

import pytest
import torch

import simplicial_attention_b200 as sa
from simplicial_attention_b200 import _lib
from simplicial_attention_b200.attention import _shape, _strides

pytestmark = pytest.mark.gpu

FORMS = {"batch": (1, None, None), "heads": (None, None, 1), "rows": (None, 1, None)}


def _operands(form, d, dtype, b=3, n=140, hq=4, hk=2):
    g = torch.Generator(device="cuda").manual_seed(d)
    mk = lambda s: torch.randn(s, device="cuda", generator=g).to(dtype)
    full = (b, n, hk, d)
    one = tuple(f or s for f, s in zip(FORMS[form], full)) + (d,)
    return mk((b, n, hq, d)), [mk(one).expand(full) for _ in range(4)], mk((b, n, hq, d))


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("d,w1,w2,dtype", [(32, 100, 9, torch.bfloat16), (64, 100, 9, torch.bfloat16), (64, 600, 9, torch.bfloat16),
                                           (64, 140, 70, torch.bfloat16), (128, 100, 9, torch.bfloat16), (64, 100, 9, torch.float32)])
def test_expanded_equals_contiguous(form, d, w1, w2, dtype):
    q, kv, dout = _operands(form, d, dtype)
    res = []
    for keys in (kv, [t.contiguous() for t in kv]):
        ins = [t.detach().requires_grad_() for t in (q, *keys)]
        out = sa.sliding_two_simplicial_attn(ins[0], ins[1:3], ins[3:5], w1=w1, w2=w2)
        k1, k2, v1, v2 = (t.detach() for t in ins[1:])
        raw, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2)
        res.append([out.detach(), raw, lse, *torch.autograd.grad(out, ins, dout), *sa.sa2_backward(q, k1, k2, v1, v2, raw, lse, dout, w1, w2)])
    assert sa.device_status() == 0
    assert all(torch.equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("form", FORMS)
def test_strides_of_zero_at_the_abi(form):
    """AUTO takes the kernels that can address them; TCGEN05 says that it cannot."""
    q, (k1, k2, v1, v2), _ = _operands(form, 64, torch.bfloat16)
    want, _ = sa.sa2_forward(q, *(t.contiguous() for t in (k1, k2, v1, v2)), 100, 9, kernel="simt")
    out, lse = torch.empty_like(q), torch.empty(3, 4, 140, device="cuda")
    for kernel, status in (("auto", 0), ("tcgen05", 2)):
        args = _lib.FwdArgs(_shape(q, k1, k2, 100, 9, 64 ** -0.5, kernel), *(t.data_ptr() for t in (q, k1, k2, v1, v2, out, lse)),
                            *(_strides(t) for t in (q, k1, k2, v1, v2, out)), torch.cuda.current_stream().cuda_stream)
        assert _lib.lib().sa2_fwd(C.byref(args)) == status
    assert torch.equal(out, want)


@pytest.mark.parametrize("d,w1,w2", [(32, 100, 9), (64, 100, 9), (64, 600, 70), (128, 100, 9)])
def test_head_first_memory(d, w1, w2):
    """Operands and output gradient stored (b, h, n, d): strides in another order, read in place."""
    q, kv, dout = _operands("batch", d, torch.bfloat16)
    plain = [t.contiguous() for t in (q, *kv, dout)]
    turned = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in plain]
    res = []
    for q, k1, k2, v1, v2, do in (plain, turned):
        out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2)
        res.append([out, lse, *sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2)])
    assert sa.device_status() == 0
    assert all(torch.equal(a, b) for a, b in zip(*res))
