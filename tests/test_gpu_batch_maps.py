"""Batches made one after another in the same device memory: the tensor maps of each lie in global memory,
where the ones of the batch before lay, and must be read anew.  One iteration against FP64; the tolerance is
that of the FP32 products after one iteration (test_gpu_split_batch)."""
import numpy as np
import pytest

from gpumlib_gb300.batch import Batch
from test_gpu_split_batch import EPS, TOL, _instance, _step64


@pytest.mark.gpu
def test_new_batch_in_the_memory_of_the_last():
    for turn in range(6):
        rng = np.random.default_rng(turn)
        insts = [_instance(int(rng.integers(60, 500)), int(rng.integers(60, 400)), int(rng.choice((4, 9, 16, 31))), 100 * turn + k)
                 for k in range(60)]
        with Batch(insts, eps=EPS) as b:
            b.run(1)
            b.synchronize()
            for k, d in enumerate(insts):
                Wg, Hg = b.get(k)
                W1, H1 = _step64(*(d[x].astype(np.float64) for x in "VWH"))
                assert np.max(np.abs(Hg - H1) / H1) <= TOL and np.max(np.abs(Wg - W1) / W1) <= 2 * TOL
