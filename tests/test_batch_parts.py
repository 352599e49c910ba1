"""How the backward is split over CTAs follows the batch: many short sequences pay neither time nor scratch for splits
that only a small batch needs, and parts of a batch that say so get the whole batch's bits."""
import ctypes as C

import pytest
import torch

import simplicial_attention_b200 as sa
from oracle import oracle as O
from simplicial_attention_b200 import _lib
from test_abi import _shape


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("b,n,hq,hk", [(128, 128, 8, 8), (64, 256, 8, 4), (256, 128, 8, 8)])
def test_scratch_of_many_short_sequences(b, n, hq, hk, d):
    """No more than one range of offsets per query tile takes: two slabs of 127 + 32 rows for 128 query rows, one partial dQ
    per window split, and dK1 / dV1 in at most two parts."""
    s = _shape(b=b, n=n, hq=hq, hk=hk, d=d, w1=512, w2=32, dtype=1)
    q, k = b * n * hq * d * 4, b * n * hk * d * 4
    assert _lib.lib().sa2_bwd_workspace_bytes(C.byref(s)) <= b * n * hq * 4 + q * 2 * 159 / 128 + 2 * q + 4 * k + 1024


def test_a_part_is_sized_as_its_whole():
    lib, s = _lib.lib(), _shape(b=2, n=128, hq=8, hk=8, w1=512, w2=32, dtype=1)
    part = lambda whole: lib.sa2_bwd_workspace_bytes_part(C.byref(s), whole)
    assert part(2) == lib.sa2_bwd_workspace_bytes(C.byref(s)) > part(128) > 0
    assert part(1) == 0 and lib.sa2_bwd_part(None, 4) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("n,hq,hk,d,w1,w2", [(128, 8, 8, 64, 64, 32), (200, 4, 1, 128, 100, 20), (150, 4, 4, 32, 150, 40), (150, 4, 2, 64, 150, 80)])
def test_parts_have_the_bits_of_the_whole(n, hq, hk, d, w1, w2):
    b = 37
    q, k1, k2, v1, v2, do = [t.cuda() for t in O.make_inputs(b, n, hq, hk, d, seed=4, dtype=torch.bfloat16)]
    out, lse = sa.sa2_forward(q, k1, k2, v1, v2, w1, w2)
    whole = sa.sa2_backward(q, k1, k2, v1, v2, out, lse, do, w1, w2)
    for s in (slice(0, 1), slice(7, 10), slice(30, 37)):
        po, pl = sa.sa2_forward(q[s], k1[s], k2[s], v1[s], v2[s], w1, w2)
        assert torch.equal(po, out[s]) and torch.equal(pl, lse[s])
        part = sa.sa2_backward(q[s], k1[s], k2[s], v1[s], v2[s], po, pl, do[s], w1, w2, whole_batch=b)
        assert all(torch.equal(x, y[s]) for x, y in zip(part, whole))
    assert sa.device_status() == 0


@pytest.mark.gpu
def test_host_pipeline_chunks_have_the_bits_of_the_whole():
    b, n, h, d = 37, 128, 8, 64
    host = [t.pin_memory() for t in O.make_inputs(b, n, h, h, d, seed=6, dtype=torch.bfloat16)]
    outs = [torch.empty_like(t).pin_memory() for t in host]
    pipe = sa.HostPipeline("cuda:0", w1=64, w2=32, chunk=3)
    pipe.run(host, outs)
    pipe.synchronize()
    dev = [t.cuda() for t in host]
    out, lse = sa.sa2_forward(*dev[:5], 64, 32)
    for got, want in zip(outs, (out, *sa.sa2_backward(*dev[:5], out, lse, dev[5], 64, 32))):
        assert torch.equal(got, want.cpu())
