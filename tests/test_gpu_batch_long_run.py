"""A long run of a batch whose instances share their launches: the same bits as many short ones, and the call
returns while the GPU is still at work."""
import time

import numpy as np
import pytest

from gpumlib_gb300.batch import Batch
from test_gpu_split_batch import _instance


@pytest.mark.gpu
@pytest.mark.parametrize("iters", [128, 129, 300])
def test_same_bits(iters):
    insts = [_instance(400 + 7 * k, 300, 16, k) for k in range(30)]
    with Batch(insts) as a, Batch(insts) as b:
        assert a.shares_launches
        a.run(iters)
        for _ in range(iters):
            b.run(1)
        for k in range(a.count):
            assert all(np.array_equal(x, y) for x, y in zip(a.get(k), b.get(k)))


@pytest.mark.gpu
def test_does_not_wait():
    insts = [_instance(1024, 512, 32, k) for k in range(300)]
    with Batch(insts) as b:
        assert b.shares_launches
        b.run(200)
        b.synchronize()
        t0 = time.perf_counter()
        b.run(2000)
        t1 = time.perf_counter()
        b.synchronize()
        t2 = time.perf_counter()
    assert t1 - t0 <= 0.5 * (t2 - t0)
