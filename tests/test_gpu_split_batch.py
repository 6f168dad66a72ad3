"""Batches whose half-steps share their launches (tiles of all instances over the SMs): against FP64 at the
edges of tiles (128 rows), chunks (64 of K), update blocks (64 rows), rank padding (16 / 32) and V strides
(n % 4), with instances on both sides of a CTA's share; repeated runs, fresh factors.

Tolerance per element after one iteration: that of the FP32 products (test_gpu_split_fp32), 1.6e-5 for H and
twice that for W; two iterations: three times the W bound."""
import numpy as np
import pytest

from gpumlib_gb300.batch import Batch

TOL = 1.6e-5
EPS = 1e-8
SHAPES = [(1024, 512, 32), (33, 40, 4), (128, 64, 16), (129, 65, 17), (127, 63, 5), (1000, 511, 31), (64, 200, 1),
          (700, 300, 8), (257, 129, 32), (130, 500, 10)]


def _instance(n, m, r, seed):
    rng = np.random.default_rng(seed)
    u = lambda a, b: rng.random((a, b), dtype=np.float32) + np.float32(0.01)  # noqa: E731
    return {"V": u(n, m), "W": u(n, r), "H": u(r, m)}


def _step64(V, W, H):
    H = H * ((W.T @ V) / (W.T @ W @ H + EPS))
    return W * ((V @ H.T) / (W @ (H @ H.T) + EPS)), H


@pytest.mark.gpu
@pytest.mark.parametrize("copies", [1, 40])
def test_against_fp64(copies):
    insts = [_instance(*s, seed=k) for k, s in enumerate(SHAPES)]
    with Batch(insts * copies, eps=EPS) as b:
        b.run(1)
        b.synchronize()
        one = [b.get(k) for k in range(b.count)]
        res = b.residuals()
        b.run(1)
        two = [b.get(k) for k in range(len(SHAPES))]
        b.reset_factors()
        b.run(1)
        again = [b.get(k) for k in range(len(SHAPES))]
    for k, d in enumerate(insts):
        V, W, H = (d[x].astype(np.float64) for x in "VWH")
        W1, H1 = _step64(V, W, H)
        for c in range(copies):  # the same instance anywhere in the batch
            Wg, Hg = one[c * len(insts) + k]
            assert np.max(np.abs(Hg - H1) / H1) <= TOL
            assert np.max(np.abs(Wg - W1) / W1) <= 2 * TOL
        Wg, Hg = one[k]
        exact = np.linalg.norm(V - Wg.astype(np.float64) @ Hg) / np.linalg.norm(V)
        assert abs(res[k] - exact) <= 1e-6 * max(1.0, exact)
        W2, H2 = _step64(V, W1, H1)
        assert np.max(np.abs(two[k][0] - W2) / W2) <= 6 * TOL
        assert np.max(np.abs(two[k][1] - H2) / H2) <= 6 * TOL
        assert np.array_equal(again[k][0], Wg) and np.array_equal(again[k][1], Hg)
