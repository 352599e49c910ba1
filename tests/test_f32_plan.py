"""Scratch of the fp32 backward on the tensor cores (head dims 32 and 64): no shape of ordinary size falls back to the scalar kernels for
want of scratch, and none takes more than a round's.  Host arithmetic only: no GPU."""
import ctypes as C
import random

import pytest

from simplicial_attention_b200 import _lib

ROUND = 256 << 20


def _plan(b, n, hq, hk, d, w1, w2):
    shape = _lib.Shape(b, n, hq, hk, d, w1, w2, 0, 0, _lib.SA2_F32, _lib.KERNELS["auto"], d ** -0.5)
    rowsums = -(-b * hq * n * 4 // 256) * 256
    return _lib.lib().sa2_kernel_launches(C.byref(shape), 1), _lib.lib().sa2_bwd_workspace_bytes(C.byref(shape)) - rowsums


# groups of query heads: the dQ slabs are one per query head and range of offsets
NAMED = [(1, 14406, 16, 2, 64, 507, 31), (1, 8085, 16, 2, 64, 425, 49), (1, 16170, 4, 1, 64, 1022, 37), (1, 3584, 8, 1, 64, 3584, 256),
         (1, 16384, 32, 1, 64, 512, 64), (1, 16384, 64, 1, 64, 512, 32), (1, 6308, 8, 1, 64, 460, 19)]


@pytest.mark.parametrize("shape", NAMED, ids=str)
def test_groups_of_query_heads(shape):
    launches, scratch = _plan(*shape)
    least = shape[2] * -(-shape[1] // 128) * (127 + shape[6]) * shape[4] * 4       # one range of offsets
    assert launches > 2
    assert scratch <= max(ROUND, least) + 4096


def test_random_shapes():
    rng = random.Random(0)
    for _ in range(3000):
        hk = rng.choice((1, 2, 3, 4, 8))
        hq = hk * rng.choice((1, 2, 4, 8))
        n = int(2 ** rng.uniform(0, 14))
        shape = (rng.randint(1, 8), n, min(hq, 16) // hk * hk or hk, hk, rng.choice((32, 64)), rng.randint(1, 1024), rng.randint(1, 64))
        launches, scratch = _plan(*shape)
        assert launches > 2, shape
        assert scratch <= ROUND + 4096, shape
