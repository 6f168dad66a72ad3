"""BF16 KL jobs whose CTAs stream many V blocks through their ring of stages: the same bits every time, with
the sample and without.  (A stage refilled before its values had been used would change some of them.)"""
import numpy as np
import pytest

import gpumlib_gb300 as g


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,r", [(4096, 2048, 128), (2049, 3000, 40), (16384, 1024, 64)])
def test_same_bits_every_time(n, m, r):
    rng = np.random.default_rng(n + r)
    V = np.asfortranarray(rng.poisson(2.0, (n, m)).astype(np.float32))
    W = np.asfortranarray(rng.random((n, r), dtype=np.float32) + np.float32(0.05))
    H = np.asfortranarray(rng.random((r, m), dtype=np.float32) + np.float32(0.05))
    got = []
    for sampled in (1, 0, 1, 0, 1):
        with g.make(1, V, W, H, eps=1e-6, precision="bf16", quality_interval=sampled) as job:
            job.Iterate(4)
            got.append((job.GetW(), job.GetH()))
    assert all(np.array_equal(w, got[0][0]) and np.array_equal(h, got[0][1]) for w, h in got)
