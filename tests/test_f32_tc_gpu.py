"""fp32 tensors on the tensor cores (head dims 32 and 64, kernel="auto"): edges of the 128-row tiles and 64-column units, splits of
heads and offsets, halos, strides, and non-finite operands.  Against the oracle in 64 bits."""
import pytest
import torch

import simplicial_attention_b200 as sa
from oracle import oracle as O
from simplicial_attention_b200 import _lib

pytestmark = pytest.mark.gpu
GRADS = ("dq", "dk1", "dk2", "dv1", "dv2")
# A logit of magnitude below 8 is off by at most half a unit in its last place, 2^-22, times log2(e) and the few sums behind it:
# every weight is within 2^-21 of itself, and so is a result in norm; twice that leaves room for the sums of the gradients.
REL = 2. ** -20

CASES = [
    # b, n, hq, hk, d, w1, w2
    (1, 1, 1, 1, 64, 1, 1),
    (1, 64, 1, 1, 64, 64, 1),          # one offset: the second softmax group has none
    (2, 127, 2, 1, 32, 63, 3),
    (1, 128, 2, 2, 32, 128, 128),      # many offset ranges of one tile
    (1, 129, 3, 3, 64, 65, 2),
    (1, 200, 8, 1, 64, 64, 5),         # heads of a group split over CTAs
    (3, 77, 6, 3, 32, 33, 77),
    (1, 333, 2, 1, 64, 700, 70),       # windows longer than the sequence
    (1, 700, 4, 4, 64, 512, 32),
]


def _norm_err(x, ref):
    ref = ref.double().cpu()
    return ((x.double().cpu() - ref).norm() / ref.norm().clamp_min(1e-3 * ref.numel() ** 0.5)).item()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%d_n%d_hq%d_hk%d_d%d_w%d_%d" % c)
def test_matches_oracle(case):
    b, n, hq, hk, d, w1, w2 = case
    ins = O.make_inputs(b, n, hq, hk, d, seed=n)
    ref = O.two_simplicial_fwd_bwd(*ins, w1, w2, dtype=torch.float64)
    q, k1, k2, v1, v2, do = (t.cuda() for t in ins)
    out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2)
    grads = sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2)
    again = sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2)
    assert sa.device_status() == 0
    assert all(torch.equal(x, y) for x, y in zip(grads, again))
    # (gradients that vanish, as with one key per row, are compared with the size of the others)
    floor = max(ref[g].norm().item() / ref[g].numel() ** 0.5 for g in GRADS)
    for name, x in (("out", out), ("lse", lse), *zip(GRADS, grads)):
        r = ref[name].double()
        err = (x.double().cpu() - r).norm().item()
        assert err <= REL * max(r.norm().item(), floor * r.numel() ** 0.5), (name, err / max(r.norm().item(), 1e-30))


@pytest.mark.parametrize("d", [32, 64])
def test_halo_and_strides(d):
    """A block of rows behind halo rows, operands as views of wider tensors, against the scalar kernels on the same."""
    g = torch.Generator(device="cuda").manual_seed(d)
    n, off1, off2, w1, w2 = 150, 90, 7, 100, 9
    wide = lambda rows, h: torch.randn(2, rows, h, 2 * d + 4, device="cuda", generator=g)[..., 4:4 + d]
    q, do = wide(n, 4), wide(n, 4)
    k1, v1, k2, v2 = wide(n + off1, 2), wide(n + off1, 2), wide(n + off2, 2), wide(n + off2, 2)
    res = []
    for kernel in ("auto", "simt"):
        out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2, kernel=kernel)
        res.append((out, lse, *sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2, kernel=kernel)))
    assert sa.device_status() == 0
    for x, y in zip(*res):
        assert (x.double() - y.double()).norm() <= 2 * REL * y.double().norm()      # either is within the bound of the exact value


@pytest.mark.parametrize("d", [32, 64])
def test_infinite_keys_weigh_nothing(d):
    """First keys of -inf against positive rows: their terms are no numbers, their logits are, and the rest is unharmed."""
    g = torch.Generator(device="cuda").manual_seed(d)
    q, k1, k2, v1, v2 = (torch.randn(1, 200, 2, d, device="cuda", generator=g) for _ in range(5))
    for t in (q, k1, k2):
        t.abs_()
    k1[:, 60:155] = -torch.inf
    out, lse = sa.sa2_forward(q, k1, k2, v1, v2, 100, 4)
    want, want_lse = sa.sa2_forward(q, k1, k2, v1, v2, 100, 4, kernel="simt")
    seen = want_lse.isfinite()                        # rows whose whole window is -inf have no answer
    assert seen.sum() >= 300 and torch.equal(lse.isfinite(), seen)
    rows = seen.transpose(1, 2)
    assert (out[rows] - want[rows]).norm() <= 2 * REL * want[rows].norm()


def _same(x, want):
    """The same NaN and infinities, and finite values within the error of either kernel."""
    assert torch.equal(x.isnan(), want.isnan())
    assert torch.equal(x.isinf(), want.isinf()) and torch.equal(x[x.isinf()], want[want.isinf()])
    fine = want.isfinite()
    assert (x[fine].double() - want[fine].double()).norm() <= 2 * REL * want[fine].double().norm()


INF = float("inf")
ONE = [(t, v) for t in range(6) for v in (INF, -INF, float("nan"), 3.395e38, 1e-39)]


@pytest.mark.parametrize("d", [32, 64])
@pytest.mark.parametrize("which,value", ONE, ids=lambda x: str(x))
def test_values_that_three_terms_are_not(which, value, d):
    """One entry that is not finite, rounds to an infinite bf16 or is below its range: outputs and gradients are those of the scalar
    kernels, also in the rows and heads that do not see it, and the other batch element's do not move."""
    g = torch.Generator(device="cuda").manual_seed(d)
    ins = [torch.randn(2, 300, 2, d, device="cuda", generator=g) for _ in range(6)]
    plain = sa.sa2_forward(*ins[:5], 64, 9)
    before = (*plain, *sa.sa2_backward(*ins[:5], *plain, ins[5], 64, 9))
    ins[which][1, 70, 1, 5] = value
    res = []
    for kernel in ("auto", "simt"):
        out, lse = sa.sa2_forward(*ins[:5], 64, 9, kernel=kernel)
        res.append((out, lse, *sa.sa2_backward(*ins[:5], out, lse, ins[5], 64, 9, kernel=kernel)))
    assert sa.device_status() == 0
    # (a logit of 1e38 is known to 1e31: the backward, which subtracts its logsumexp, has no answer to compare)
    compared = 2 if which < 3 and value == 3.395e38 else 7
    for x, want, was in list(zip(*res, before))[:compared]:
        _same(x, want)
        assert torch.equal(x[0], was[0])


@pytest.mark.parametrize("factors", [(1, 1, 1, 1e-36, 1, 1), (1, 1, 1, 1, 1, 1e-36), (1e-18, 1e36, 1e-18, 1, 1, 1), (1e-20, 1, 1e-15, 1, 1, 1),
                                     (1, 1, 1, 1e30, 1, 1), (1, 1, 1, 1, 1, 1e30)], ids=str)
def test_tiny_and_large_operands_keep_their_bits(factors):
    """Operands whose second and third terms would leave bf16's range, and sums that would leave fp32's."""
    g = torch.Generator(device="cuda").manual_seed(1)
    ins = [f * torch.randn(1, 200, 2, 64, device="cuda", generator=g) for f in factors]
    res = []
    for kernel in ("auto", "simt"):
        out, lse = sa.sa2_forward(*ins[:5], 100, 4, kernel=kernel)
        res.append((out, lse, *sa.sa2_backward(*ins[:5], out, lse, ins[5], 100, 4, kernel=kernel)))
    assert sa.device_status() == 0
    for x, want in zip(*res):
        _same(x, want)


def test_parts_of_a_backward_do_odd_values_too():
    """The row sums clear the marks, either part of the backward does what it has marked."""
    g = torch.Generator(device="cuda").manual_seed(2)
    ins = [torch.randn(2, 200, 2, 64, device="cuda", generator=g) for _ in range(6)]
    ins[4][1, 50, 0, 3] = INF
    out, lse = sa.sa2_forward(*ins[:5], 100, 4)
    whole = sa.sa2_backward(*ins[:5], out, lse, ins[5], 100, 4)
    call = sa.BackwardCall(*ins[:5], out, lse, ins[5], 100, 4)
    for phase in (_lib.BWD_ROWSUM, _lib.BWD_K1, _lib.BWD_Q):
        call.launch(phase)
    for x, want in zip(call.grads, whole):
        assert torch.equal(x.nan_to_num(7.), want.nan_to_num(7.)) and torch.equal(x.isnan(), want.isnan())


def test_scratch_rounds():
    """A batch whose scratch passes the limit of a round goes through it in several; an element alone does in one."""
    b, n = 16, 700
    shape = _lib.Shape(b, n, 8, 8, 64, n, n, 0, 0, 0, 0, 0.125)
    assert _lib.lib().sa2_bwd_workspace_bytes(shape) <= (256 << 20) + b * n * 8 * 4 + 1024
    assert _lib.lib().sa2_kernel_launches(shape, 1) > 4
    g = torch.Generator(device="cuda").manual_seed(0)
    ins = [torch.randn(b, n, 8, 64, device="cuda", generator=g) for _ in range(6)]
    out, lse = sa.sa2_forward(*ins[:5], n, n)
    whole = sa.sa2_backward(*ins[:5], out, lse, ins[5], n, n)
    one = sa.sa2_backward(*(t[15:] for t in ins[:5]), out[15:], lse[15:], ins[5][15:], n, n)
    assert sa.device_status() == 0
    for x, y in zip(whole, one):
        assert (x[15:].double() - y.double()).norm() <= 2 * REL * y.double().norm()
