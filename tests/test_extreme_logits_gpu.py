"""Logits at the ends of their range: -inf beside finite ones."""
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
