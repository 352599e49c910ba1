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


@pytest.mark.parametrize("b,n,w2", [(1, 4096, 4096), (1, 1024, 1024), (64, 1024, 64), (8, 190, 190)])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_scratch_of_long_second_windows_is_bounded(b, n, w2, d):
    """Row sums, the partials of dK1 / dV1 (at most 16 of each), and 1 GiB for the ranges of offsets; 256 MiB where a batch
    is cut into rounds."""
    rows, tensor = b * 8 * n * 4, b * n * 8 * d * 4
    need = _lib.lib().sa2_bwd_workspace_bytes(C.byref(_shape(b=b, n=n, hq=8, hk=8, d=d, w1=n, w2=w2, dtype=1)))
    assert need <= rows + 16 * 2 * tensor + ((256 if b > 1 else 1024) << 20) + 1024


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
