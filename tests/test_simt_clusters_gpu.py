"""The fp32 kernels where their offsets are split over clusters of one to eight CTAs and over the two groups of a
CTA: fewer offsets than groups, remainders, second-key windows longer than the sequence, and every head dim."""
import pytest
import torch

from oracle import oracle as O
from test_parity_gpu import FP32_REL, GRADS, run_ours
from util import NAMES, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    # b, n, hq, hk, d, w1, w2
    (1, 64, 1, 1, 64, 64, 1),        # one offset: the second group has none
    (1, 65, 1, 1, 32, 20, 17),       # one row in the second tile, remainders in every rank
    (2, 128, 2, 1, 32, 128, 128),    # eight CTAs per tile
    (1, 100, 3, 1, 128, 30, 37),     # one group per CTA
    (1, 20, 1, 1, 64, 64, 64),       # windows longer than the sequence
    (1, 700, 8, 8, 32, 33, 5),       # enough tiles for one CTA each
], ids=lambda c: "b%d_n%d_hq%d_hk%d_d%d_w%d_%d" % c)
def test_matches_oracle(case):
    b, n, hq, hk, d, w1, w2 = case
    ins = O.make_inputs(b, n, hq, hk, d, seed=n)
    ref = O.two_simplicial_fwd_bwd(*ins, w1, w2, dtype=torch.float64)
    r = run_ours(*ins, w1, w2)
    floor = 0.05 * max(ref[k].abs().max().item() for k in GRADS)
    for k in NAMES + ("lse",):
        assert rel_err(r[k], ref[k], floor) <= FP32_REL, (k, rel_err(r[k], ref[k], floor))
