"""Windows longer than the sequence select the pairs of a window as long as the sequence: same scratch, same bits.  The
longest is the largest int32, a caller's way to say "no window"."""
import ctypes as C

import pytest
import torch

import simplicial_attention_b200 as sa
from oracle import oracle as O
from test_abi import _shape
from simplicial_attention_b200 import _lib

LONGEST = 2 ** 31 - 1


@pytest.mark.parametrize("off", [0, 70])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("w1,w2", [(LONGEST, LONGEST), (LONGEST, 32), (2 ** 20, 2 ** 20), (200, LONGEST)])
def test_scratch_is_that_of_the_sequence(w1, w2, d, off):
    def need(a, b):
        return _lib.lib().sa2_bwd_workspace_bytes(C.byref(_shape(b=8, n=128, hq=8, hk=4, d=d, w1=a, w2=b, off1=off, off2=off, dtype=1)))

    assert need(w1, w2) == need(min(w1, 128 + off), min(w2, 128 + off))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_longest_window_equals_full_causal(d, dtype):
    n, long = 100, 1024
    q, k1, k2, v1, v2, do = [t.cuda() for t in O.make_inputs(2, n, 4, 2, d, seed=d, dtype=dtype)]
    res = []
    for w1, w2 in ((LONGEST, LONGEST), (long, long)):
        out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2)
        res.append([out, lse, *sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2)])
    assert sa.device_status() == 0
    for a, b in zip(*res):
        assert torch.equal(a, b) and a.isfinite().all()
