"""The relative residual at the ends of FP32's range, by the tensor-core kernel (32768 elements and more) and the
FP32 one: V = s V1 and W H = s W1 H1 have the residual of V1 and W1 H1 whatever the power of two s is, which moves no
bit of V, W or H.  W H is within 2^-21 of its value either way: 1e-6 (the residual itself is about 0.5).
An infinity or NaN in V is no perfect fit."""
import numpy as np
import pytest

import gpumlib_gb300 as g

SHAPES = [(256, 300, 20), (90, 70, 8), (515, 129, 100)]


def _inputs(n, m, r, scale):
    rng = np.random.default_rng(n + r)
    V = rng.random((n, m), dtype=np.float32)
    V[rng.random((n, m)) < 0.3] = 0
    V[:, 5] = 0  # rows of sixteen zeros
    W, H = rng.random((n, r), dtype=np.float32), rng.random((r, m), dtype=np.float32) * np.float32(1.0 / r)
    H[:, 5] = 0
    return V * np.float32(2.0 ** scale), W * np.float32(2.0 ** (scale // 2)), H * np.float32(2.0 ** (scale - scale // 2))


def _residual(V, W, H, precision):
    with g.make(0, V, W, H, precision=precision, quality_interval=0) as job:
        return job.Residual()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("scale", [0, 40, 52, 66, 100, -36, -44, -70, -76, -90, -100])
@pytest.mark.parametrize("n,m,r", SHAPES)
def test_scaled(n, m, r, scale, precision):
    V, W, H = _inputs(n, m, r, scale)
    v, wh = V.astype(np.float64), W.astype(np.float64) @ H
    assert abs(_residual(V, W, H, precision) - np.linalg.norm(v - wh) / np.linalg.norm(v)) <= 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("n,m,r", SHAPES)
def test_not_finite(n, m, r, bad):
    V, W, H = _inputs(n, m, r, 0)
    V[n - 1, m - 1] = bad
    assert np.isnan(_residual(V, W, H, "fp32"))


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,r", SHAPES)
def test_zero_matrix(n, m, r):
    V, W, H = _inputs(n, m, r, 0)
    assert _residual(np.zeros_like(V), W, H, "fp32") == 0.0
