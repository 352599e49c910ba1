"""bf16 shapes whose arithmetic is that of fp32 (head dim 32, long first windows at head dim 64, long second windows):
only the inputs and the results are rounded to bf16.  Against the oracle in 64 bits."""
import ctypes as C

import pytest
import torch

import simplicial_attention_b200 as sa
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FORWARD = [
    # b, n, hq, hk, d, w1, w2
    (1, 1, 1, 1, 32, 4, 2),
    (2, 129, 4, 2, 32, 70, 5),        # odd number of sweeps, one row in the last tile
    (1, 300, 2, 1, 32, 300, 33),      # window from global memory, grouped-query heads
    (1, 200, 2, 2, 64, 514, 16),      # the shortest long window, longer than the sequence
    (1, 1100, 1, 1, 64, 1024, 9),     # ring of units
]


@pytest.mark.parametrize("case", FORWARD, ids=lambda c: "b%d_n%d_hq%d_hk%d_d%d_w%d_%d" % c)
def test_forward(case):
    b, n, hq, hk, d, w1, w2 = case
    ins = O.make_inputs(b, n, hq, hk, d, seed=n + w2, dtype=torch.bfloat16)
    ref, ref_lse = O.two_simplicial_fwd(*[t.double() for t in ins[:5]], w1, w2)
    out, lse = sa.sa2_forward(*[t.cuda() for t in ins[:5]], w1, w2)
    assert sa.device_status() == 0
    # sums of fp32 terms, exp2 to 2^-22 per logit: 1e-5 on logits of up to about 16
    assert (lse.double().cpu() - ref_lse).abs().max().item() <= 1e-5
    # half a unit of bf16, and 16-bit probabilities against values of about 4: 2^-17 * 4 * 4 / rms
    over = (out.double().cpu() - ref).abs() - ref.abs() * 2 ** -8
    assert over.max().item() <= 2e-4, over.max().item()


def test_generation_row():
    """One new row behind full windows."""
    w1, w2 = 600, 20
    ins = O.make_inputs(2, w1, 4, 2, 64, seed=3, dtype=torch.bfloat16)
    ref, ref_lse = O.two_simplicial_fwd(*[t.double() for t in ins[:5]], w1, w2)
    q, k1, k2, v1, v2 = [t.cuda() for t in ins[:5]]
    s = w1 - 1
    out, lse = sa.sa2_forward(q[:, s:], k1, k2[:, s - w2 + 1:], v1, v2[:, s - w2 + 1:], w1, w2)
    assert sa.device_status() == 0
    assert (lse.double().cpu() - ref_lse[:, :, s:]).abs().max().item() <= 1e-5
    over = (out.double().cpu() - ref[:, s:]).abs() - ref[:, s:].abs() * 2 ** -8
    assert over.max().item() <= 2e-4, over.max().item()


BACKWARD = [
    # b, n, hq, hk, w1, w2
    (1, 40, 1, 1, 40, 40),            # one tile, offset ranges that start past the first rows
    (2, 129, 4, 2, 70, 5),            # one row in the last tile
    (1, 300, 4, 1, 200, 33),          # four heads per key head, second-key rows from global memory
    (1, 700, 2, 2, 512, 9),           # window splits
]


@pytest.mark.parametrize("case", BACKWARD, ids=lambda c: "b%d_n%d_hq%d_hk%d_w%d_%d" % c)
def test_backward_head_dim_32(case):
    """Gradients of bf16 operands in bf16, next to those of the fp32 kernels for the same saved output: both are off
    from 64 bits by their rounding to bf16 and by that of the saved output, and by nothing else that shows."""
    b, n, hq, hk, w1, w2 = case
    ins = O.make_inputs(b, n, hq, hk, 32, seed=n + w2, dtype=torch.bfloat16)
    ref = O.two_simplicial_fwd_bwd(*[t.double() for t in ins], w1, w2, dtype=torch.float64)
    q, k1, k2, v1, v2, do = [t.cuda() for t in ins]
    out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2, kernel="simt")
    got, base = (sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2, kernel=k) for k in ("auto", "simt"))
    fine, base_fine = (sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2, kernel=k, grad_dtype=torch.float32) for k in ("tcgen05", "simt"))
    assert sa.device_status() == 0
    for i, name in enumerate(("dq", "dk1", "dk2", "dv1", "dv2")):
        r = ref[name]
        err = lambda x: ((x.double().cpu() - r).norm() / r.norm()).item()
        assert err(got[i]) <= 1.01 * err(base[i]) + 2e-5, (name, err(got[i]), err(base[i]))
        # 16-bit P and G in fp32 sums
        assert (fine[i] - base_fine[i]).norm() <= 2e-5 * base_fine[i].norm(), name


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("n,w1,w2", [(150, 150, 150), (90, 40, 57), (30, 20, 400), (400, 300, 60)])
def test_long_second_window(n, w1, w2, d):
    """dq, dk2 and dv2 are as far from 64 bits as those of the fp32 kernels, also where the sequence is shorter than the
    window; in fp32 they are those of the fp32 kernels."""
    ins = O.make_inputs(2, n, 2, 1, d, seed=n + d, dtype=torch.bfloat16)
    ref = O.two_simplicial_fwd_bwd(*[t.double() for t in ins], w1, w2, dtype=torch.float64)
    q, k1, k2, v1, v2, do = [t.cuda() for t in ins]
    out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2, kernel="simt")
    got, base = (sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2, kernel=k) for k in ("auto", "simt"))
    fine, same, base_fine = (sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2, kernel=k, grad_dtype=torch.float32)
                             for k in ("tcgen05", "auto", "simt"))
    assert sa.device_status() == 0
    for i, name in ((0, "dq"), (2, "dk2"), (4, "dv2")):
        err = lambda x: ((x.double().cpu() - ref[name]).norm() / ref[name].norm()).item()
        assert err(got[i]) <= 1.01 * err(base[i]) + 2e-5, (name, err(got[i]), err(base[i]))
        assert (fine[i] - base_fine[i]).norm() <= 2e-5 * base_fine[i].norm(), name       # 16-bit P and G in fp32 sums
        assert torch.equal(same[i], base_fine[i])


def test_long_second_window_in_rounds():
    """More batch elements than the scratch takes at a time."""
    b, n, w = 20, 300, 300
    q, k1, k2, v1, v2, do = [t.cuda() for t in O.make_inputs(b, n, 4, 2, 64, seed=2, dtype=torch.bfloat16)]
    out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w, w)
    call = sa.attention.BackwardCall(q, k1, k2, v1, v2, out, lse, do, w, w, grad_dtype=torch.float32, kernel="tcgen05")
    shape = call.args.shape
    assert sa._lib.lib().sa2_kernel_launches(C.byref(shape), 1) > 4
    got, base = call.launch(), sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w, w, grad_dtype=torch.float32, kernel="simt")
    assert sa.device_status() == 0
    for i in (0, 2, 4):
        e = (got[i] - base[i]).flatten(1).norm(dim=1) / base[i].flatten(1).norm(dim=1)
        assert e.max().item() <= 2e-5
    for i in (1, 3):
        assert (got[i] - base[i]).norm() <= 1e-2 * base[i].norm()
