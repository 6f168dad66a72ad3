"""Infinities and NaN in the factors and sums of FP32 jobs: what FP32 multiply-adds make of them, element by
element.  Where the result is finite it is that of FP64 within the bound of one iteration (test_gpu_split_fp32);
where not, the same of +inf, -inf and NaN."""
import time

import numpy as np
import pytest
import torch

import gpumlib_gb300 as g
from gpumlib_gb300 import _native
from test_gpu_device_factors import _factors
from test_gpu_split_fp32 import EPS, TOL, _inputs, _step64

SHAPES = [(150, 200, 20), (70, 300, 50), (300, 130, 100)]


def _same(got, want, tol):
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(np.isinf(got), inf) and np.array_equal(got[inf], want[inf])
    ok = np.isfinite(want)
    assert np.all(np.abs(got[ok] - want[ok]) <= tol * np.abs(want[ok]))


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("where", ["V", "W", "H"])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("n,m,r", SHAPES)
def test_one_step(n, m, r, bad, where, rule):
    V, W, H = _inputs(n, m, r, n)
    W[::3] = 0.5  # exact in one part: its other parts are zero
    {"V": V, "W": W, "H": H}[where][-1, 3] = bad
    with g.make(rule, V, W, H, eps=EPS, quality_interval=0) as job:
        job.DoIteration(False)
        Hg = job.GetH()
    with np.errstate(all="ignore"):
        _, He = _step64(rule, V, W, H)
    _same(Hg, He, TOL)


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,r", SHAPES)
def test_infinity_in_the_w_step(n, m, r):
    V, W, H = _inputs(n, m, r, n)
    V[5, 7] = np.inf
    with g.make(4, V, W, H, eps=EPS, quality_interval=0) as job:  # the rule without an H-step
        job.DoIteration()
        Wg = job.GetW()
    assert np.isposinf(Wg[5]).all() and np.isfinite(np.delete(Wg, 5, axis=0)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])
def test_infinite_quality(rule):
    """eps = 0 and rows of W that become zero: the sample holds V log10(0) = -inf."""
    V, W, H = _inputs(260, 300, 24, 1)
    with g.make(rule, V, W, H, eps=0.0, quality_interval=1) as job:
        dW, _ = _factors(job)
        job.Iterate(5)
        job.Synchronize()
        assert np.isfinite(job.QualityImprovement())
        dW[:, 3] = 0.0
        torch.cuda.synchronize()
        _native.check(_native.load().gpunmf_factors_changed(job._h))
        job.Iterate(1)  # takes the sample of the zero row
        job.Iterate(1)  # reads it
        assert np.isneginf(job.QualityImprovement())


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_no_crawl(rule, bad):
    """A whole row of V that is not finite, and the iterations after it: no more than a hundred times what they take
    on finite data (the sums formed again are one thread's each)."""
    V, W, H = _inputs(2048, 1536, 64, 2)
    times = {}
    for name in ("warm", "finite", "bad"):
        if name == "bad":
            V[11] = bad
        with g.make(rule, V, W, H, eps=EPS, quality_interval=1) as job:
            t0 = time.perf_counter()
            job.Iterate(10)
            job.Synchronize()
            times[name] = time.perf_counter() - t0
    assert times["bad"] <= 100 * times["finite"]
