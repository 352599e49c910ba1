"""GPU parity of the tensor-core backward where its offsets are split over CTAs: clusters of one to eight key-tile CTAs,
query tiles in several offset ranges, ranges without work at the start of a sequence, second-key windows longer than
a CTA's accumulators or than the sequence, and every head dim.  Gradients in fp32 against the fp32 kernels (themselves
held to 1e-4 against the oracle) on the same bf16 tensors and saved outputs."""
import pytest
import torch

import simplicial_attention_b200 as sa
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [
    # b, n, hq, hk, w1, w2
    (1, 40, 1, 1, 40, 40),         # one tile; ranges that start past the first rows
    (2, 128, 4, 4, 64, 32),        # few tiles: many ranges of few offsets
    (1, 300, 4, 1, 200, 9),        # remainders: nine offsets over the ranks, four heads per key head
    (1, 257, 2, 2, 100, 33),       # one row in the last tile
    (1, 150, 1, 1, 150, 150),      # more offsets than a CTA's accumulators hold
    (1, 100, 2, 1, 30, 400),       # second-key window longer than the sequence
    (1, 900, 2, 2, 800, 5),        # three window splits times offset splits
    (8, 700, 8, 8, 64, 3),         # enough tiles for one range each
]


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%d_n%d_hq%d_hk%d_w%d_%d" % c)
def test_split_backward_matches_fp32_kernels(case, d):
    b, n, hq, hk, w1, w2 = case
    q, k1, k2, v1, v2, do = [t.cuda() for t in O.make_inputs(b, n, hq, hk, d, seed=n + w2 + d, dtype=torch.bfloat16)]
    out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2, kernel="simt")
    ref, got = (sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2, kernel=k, grad_dtype=torch.float32) for k in ("simt", "tcgen05"))
    assert sa.device_status() == 0
    for name, a, r in zip(("dq", "dk1", "dk2", "dv1", "dv2"), got, ref):
        assert (a - r).norm() <= 1e-2 * r.norm(), (name, ((a - r).norm() / r.norm()).item())
