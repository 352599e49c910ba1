"""The one-token kernel of generation (norms, cache hand-over and attention in one launch) and the projections of up to 64 rows:
remainders of keys, offsets and heads, short and over-long caches, and the shapes that go elsewhere.  Against the same module
called module by module."""
import pytest
import torch

import simplicial_attention_b200 as sa

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
