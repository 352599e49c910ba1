"""dQ, dK2 and dV2 on tiles of 64 query rows times two offsets, and of 128 rows and one: lengths around a tile, odd numbers of
offsets, a window of one unit more than a CTA holds, ranges of offsets, halos.  Against the fp32 kernels on the same bf16 tensors."""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import simplicial_attention_b200 as sa

pytestmark = pytest.mark.gpu
# A_e, B_e, P and G are rounded to 8 bits (2^-9 each, root of their squares 2^-8), a result in bf16 to another 2^-9: 5e-3 where the
# errors of many pairs average, twice that and room where a row has few.
REL = 2e-2

CASES = [
    # b, n, hq, hk, d, w1, w2, off
    (1, 63, 1, 1, 64, 20, 1, 0),          # one offset: the odd rows have none
    (2, 64, 2, 1, 64, 64, 2, 0),
    (1, 65, 2, 2, 64, 30, 3, 0),          # one row in the second tile
    (2, 127, 4, 2, 32, 64, 5, 0),
    (1, 130, 2, 2, 128, 65, 31, 0),
    (1, 200, 1, 1, 128, 128, 1, 0),
    (1, 700, 4, 1, 64, 514, 33, 0),       # ten units: two splits of the window
    (1, 300, 2, 2, 64, 300, 120, 0),      # three ranges of offsets, with rests
    (1, 150, 2, 1, 64, 100, 9, 70),       # halo rows in front
    (1, 150, 2, 1, 128, 100, 9, 70),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%d_n%d_hq%d_hk%d_d%d_w%d_%d_off%d" % c)
def test_matches_the_fp32_kernels(case):
    b, n, hq, hk, d, w1, w2, off = case
    g = torch.Generator(device="cuda").manual_seed(n + d)
    rand = lambda rows, h: torch.randn(b, rows, h, d, device="cuda", generator=g).to(torch.bfloat16)
    q, do, keys = rand(n, hq), rand(n, hq), [rand(n + off, hk) for _ in range(4)]
    out, lse = sa.sa2_forward(q, *keys, w1, w2)
    got, again = (sa.sa2_backward(q, *keys, out, lse, do, w1, w2, grad_dtype=torch.float32, kernel="tcgen05") for _ in range(2))
    want = sa.sa2_backward(q, *keys, out, lse, do, w1, w2, grad_dtype=torch.float32, kernel="simt")
    assert sa.device_status() == 0
    for x, (a, r, w) in enumerate(zip(got, again, want)):
        assert torch.equal(a, r)
        assert (a - w).norm() <= REL * w.norm(), (x, ((a - w).norm() / w.norm()).item())


# shapes that run on tiles of 128 rows and one offset
ROWS = [
    (40, 128, 8, 2, 64, 512, 5, 0),
    (32, 100, 8, 8, 32, 100, 3, 0),
    (12, 450, 8, 4, 64, 200, 1, 0),       # one sweep
    (6, 700, 8, 2, 64, 64, 7, 0),
    (20, 128, 8, 2, 64, 128, 63, 0),      # two ranges of offsets, with rests
    (18, 200, 8, 4, 64, 60, 11, 70),      # halo rows in front
    (18, 200, 8, 4, 32, 60, 11, 70),
]


@pytest.mark.parametrize("case", ROWS, ids=lambda c: "b%d_n%d_hq%d_hk%d_d%d_w%d_%d_off%d" % c)
def test_short_windows_take_tiles_of_128_rows(case):
    test_matches_the_fp32_kernels(case)
    b, n, hq, hk, d, w1, w2, off = case
    q, *keys = [torch.randn(b, rows, h, d, device="cuda", dtype=torch.bfloat16) for rows, h in ((n, hq),) + ((n + off, hk),) * 4]
    out, lse = sa.sa2_forward(q, *keys, w1, w2)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        sa.sa2_backward(q, *keys, out, lse, q, w1, w2)
        torch.cuda.synchronize()
    names = [e.key for e in p.key_averages()]
    assert any("bwd_q_kernel<" in k and "false>" in k for k in names), names
