"""Logits at the ends of their range: -inf and NaN beside finite ones, steep climbs, negative and zero scales."""
import pytest
import torch

import simplicial_attention_b200 as sa

pytestmark = pytest.mark.gpu


def _reference(q, k1, k2, v1, v2, w1, w2):
    """64-bit softmax over every (j, k) pair; a logit beyond fp32 counts as infinite, as it does in fp32 products."""
    q, k1, k2, v1, v2 = (t.double().transpose(1, 2) for t in (q, k1, k2, v1, v2))
    n, d = q.shape[-2:]
    i = torch.arange(n, device=q.device)
    near = lambda w: ((i[:, None] - i >= 0) & (i[:, None] - i < w))
    s = torch.einsum("bhic,bhjc,bhkc->bhijk", q, k1, k2) * d ** -0.5
    s = torch.where(s < -3.4e38, -torch.inf, s).masked_fill(~(near(w1)[:, :, None] & near(w2)[:, None, :]), -torch.inf)
    p = s.flatten(-2).softmax(-1).view_as(s)
    return torch.einsum("bhijk,bhjc,bhkc->bhic", p, v1, v2).transpose(1, 2)


def _operands(d, dtype, n=200, h=2):
    g = torch.Generator(device="cuda").manual_seed(d)
    return [torch.randn(1, n, h, d, device="cuda", generator=g).to(dtype) for _ in range(5)]


@pytest.mark.parametrize("d", [32, 64, 128])
def test_logits_of_minus_infinity_weigh_nothing_fp32(d):
    """A stretch of first keys as long as a tile whose every logit is -inf; every row also sees finite ones."""
    w1, w2 = 100, 4
    ins = _operands(d, torch.float32)
    for t in ins[:3]:
        t.abs_()
    ins[1][:, 60:155] = -3e38
    out, lse = sa.sa2_forward(*ins, w1, w2)
    ref = _reference(*ins, w1, w2)
    seen = ref.isfinite().all(-1).all(-1)[0]           # rows whose whole window is -inf have no answer
    assert seen.sum() >= 150
    assert lse[:, :, seen].isfinite().all()
    assert (out[:, seen] - ref[:, seen]).abs().max().item() <= 1e-4 * ref[:, seen].abs().max().item()


@pytest.mark.parametrize("d", [32, 64, 128])
def test_rising_logits_with_large_values_fp32(d):
    """Logits that climb by 60 over the window next to values of 1e22: the partial sums stay inside fp32."""
    w1, w2 = 200, 3
    q, k1, k2, v1, v2 = _operands(d, torch.float32)
    q.fill_(1.)
    k2.fill_(1.)
    k1[:] = (torch.arange(200, device="cuda") * (0.3 * d ** -0.5)).view(1, -1, 1, 1)
    v1 *= 1e22
    out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2)
    ref = _reference(q, k1, k2, v1, v2, w1, w2)
    assert (out - ref).abs().max().item() <= 1e-4 * ref.abs().max().item()


@pytest.mark.parametrize("sign", [1., -1.])
@pytest.mark.parametrize("size", [300., 700., 3000.])
@pytest.mark.parametrize("d", [32, 64])
def test_large_finite_logits_fp32(d, size, sign):
    """Logits of 1e8 to 1e11, all of one sign: a row is its largest logit's value, far ahead of what either kernel's logits are off by
    (a few units in the last place), so that the weights are 0 and 1 and a result is v1 * v2 to the last bits."""
    ins = _operands(d, torch.float32)
    for t in ins[:3]:
        t.abs_().mul_(size)
    out, lse = sa.sa2_forward(*ins, 100, 4, scale=sign * d ** -0.5)
    want, want_lse = sa.sa2_forward(*ins, 100, 4, scale=sign * d ** -0.5, kernel="simt")
    assert sa.device_status() == 0
    assert want.isfinite().all() and out.isfinite().all() and lse.isfinite().all()
    assert (out - want).norm() <= 2 ** -20 * want.norm()
    assert (lse - want_lse).norm() <= 2 ** -20 * want_lse.norm()


BF16 = [(32, 100), (64, 100), (64, 600), (128, 100)]


@pytest.mark.parametrize("d,w1", BF16)
def test_logits_of_minus_infinity_weigh_nothing_bf16(d, w1):
    ins = _operands(d, torch.bfloat16)
    for t in ins[:3]:
        t.abs_()
    ins[1][:, 60:155] = -3e38
    out, lse = sa.sa2_forward(*ins, w1, 4)
    ref = _reference(*ins, w1, 4)
    assert sa.device_status() == 0
    seen = ref.isfinite().all(-1).all(-1)[0]
    assert seen.sum() >= 150 and lse[:, :, seen].isfinite().all()
    assert (out[:, seen].double() - ref[:, seen]).norm() <= 1e-2 * ref[:, seen].norm()


@pytest.mark.parametrize("d,w1", BF16)
def test_nan_stays_where_it_is_seen_bf16(d, w1):
    """A NaN key reaches the rows whose window holds it and no others."""
    ins = _operands(d, torch.bfloat16)
    ins[1][:, 70, 1] = float("nan")
    out, lse = sa.sa2_forward(*ins, w1, 4)
    assert sa.device_status() == 0
    want = torch.zeros(200, dtype=torch.bool, device="cuda")
    want[70:70 + w1] = True
    assert out[0, :, 0].isfinite().all() and lse[0, 0].isfinite().all()
    assert torch.equal(out[0, :, 1].isnan().all(-1), want) and torch.equal(out[0, :, 1].isnan().any(-1), want)


@pytest.mark.parametrize("scale", [-0.125, -3.])
@pytest.mark.parametrize("d,w1", BF16)
def test_negative_scale_bf16(d, w1, scale):
    """Rounded products put a logit off by at most |scale| * 2^-9 * sum_c |q k1 k2|, a sum of about d / 2 and below d here;
    their root mean square, |scale| * 2^-9 * sqrt(d / 3) <= 0.04, bounds the output's relative error with room."""
    ins = _operands(d, torch.bfloat16)
    out, lse = sa.sa2_forward(*ins, w1, 4, scale=scale)
    want, want_lse = sa.sa2_forward(*ins, w1, 4, scale=scale, kernel="simt")
    assert sa.device_status() == 0
    assert (lse - want_lse).abs().max().item() <= -scale * 2 ** -9 * d
    assert (out.float() - want.float()).norm() <= (1e-2 if scale > -1 else 0.1) * want.float().norm()


@pytest.mark.parametrize("d", [32, 64, 128])
def test_zero_scale_bf16(d):
    """Uniform weights: dq, dk1 and dk2 are zero, dv1 and dv2 are those of the fp32 kernels."""
    ins = _operands(d, torch.bfloat16)
    out, lse = sa.sa2_forward(*ins, 100, 4, scale=0.)
    got, want = (sa.sa2_backward(*ins, out, lse, ins[0], 100, 4, scale=0., kernel=k) for k in ("auto", "simt"))
    assert sa.device_status() == 0
    for a, b in zip(got, want):
        assert a.isfinite().all() and (a.float() - b.float()).norm() <= 1e-2 * b.float().norm()
