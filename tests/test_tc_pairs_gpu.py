"""GPU parity of the forward kernel at the edges of its tiles of (query row, second-key offset) pairs: tiles of 8
to 64 query rows, windows that are resident and windows that stream, staged and unstaged second-key rows, head
dims 32 and 64, and generation (few new rows behind a halo)."""
import pytest
import torch

import simplicial_attention_b200 as sa
from oracle import oracle as O
from util import max_abs

pytestmark = pytest.mark.gpu

CASES = [
    # b, n, hq, hk, d, w1, w2
    (1, 1, 1, 1, 64, 4, 2),            # one row, one key
    (1, 33, 2, 1, 32, 40, 3),          # head dim 32, one offset more than a tile of two per sweep
    (2, 300, 4, 2, 32, 100, 17),
    (1, 700, 2, 2, 32, 700, 65),       # head dim 32, streamed window, second-key rows from global memory
    (1, 1500, 2, 1, 64, 1024, 16),     # window longer than shared memory
    (1, 1200, 1, 1, 64, 705, 9),       # ring of units, odd number of sweeps in the small tiles
    (1, 190, 2, 2, 64, 190, 190),      # full causal attention: 190 offsets
    (8, 640, 16, 16, 64, 64, 8),       # enough tiles for 64 query rows each, two units per sweep
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%d_n%d_hq%d_hk%d_d%d_w%d_%d" % c)
def test_forward_matches_oracle(case):
    b, n, hq, hk, d, w1, w2 = case
    ins = O.make_inputs(b, n, hq, hk, d, seed=n + w2, dtype=torch.bfloat16)
    ref_out, ref_lse = O.two_simplicial_fwd(*[t.float() for t in ins[:5]], w1, w2)
    out, lse = sa.sa2_forward(*[t.cuda() for t in ins[:5]], w1, w2, kernel="tcgen05")
    assert sa.device_status() == 0
    err = ((out.float().cpu() - ref_out).abs() - ref_out.abs() / 256).clamp_min(0).max().item()   # less the rounding of out itself
    assert err <= 2e-2, err
    assert max_abs(lse, ref_lse) <= 2e-2


@pytest.mark.parametrize("n,w1,w2", [(1, 512, 32), (1, 64, 8), (3, 200, 33), (20, 513, 16)])
def test_generation_rows_match_the_whole_sequence(n, w1, w2):
    b, total, hq, hk, d = 3, 600, 4, 2, 64
    q, k1, k2, v1, v2, _ = [t.cuda() for t in O.make_inputs(b, total, hq, hk, d, seed=w1, dtype=torch.bfloat16)]
    out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2, kernel="simt")
    s = total - n
    part, plse = sa.sa2_forward(q[:, s:], k1[:, s - w1 + 1:], k2[:, s - w2 + 1:], v1[:, s - w1 + 1:], v2[:, s - w2 + 1:], w1, w2,
                                kernel="tcgen05")
    assert sa.device_status() == 0
    assert max_abs(part, out[:, s:]) <= 2e-2 and max_abs(plse, lse[:, :, s:]) <= 2e-2
