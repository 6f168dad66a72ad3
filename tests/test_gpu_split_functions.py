"""The FP32 kernels' own logarithm and quotient against CUDA's operations' rounding.

Logarithm: a 1 x 1 job whose W H is x exactly (W = 1) has the quality V log10(x) - x; with V = 2^50 the x is below the
result's last place.  The polynomial's 1.9 units in the last place and four roundings of half a unit (product,
difference, read-back, improvement) make 4 units of 2^-23.
Quotient: with W = 1 x 1 of 1, H = a power of two, a KL step is H (V / (H + eps)), the quotient scaled: within one unit of the
FP32 division (half for the correctly rounded quotient's last bit, and what S is expected to be low by, 0.7 * 2^-24)."""
import numpy as np
import pytest
import torch

import gpumlib_gb300 as g
from gpumlib_gb300 import _native
from test_gpu_device_factors import _factors


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])  # the kernel of its own, and the one that rides on the H-step
def test_log10(rule):
    one = np.ones((1, 1), dtype=np.float32, order="F")
    big = np.float32(2.0 ** 50)
    rng = np.random.default_rng(0)
    x = np.concatenate([2.0 ** rng.uniform(-20, 20, 150), 1 + rng.uniform(-0.3, 0.45, 150), 1 + 2.0 ** rng.uniform(-22, -3, 60),
                        2.0 ** np.arange(-20, 21), np.sqrt(0.5) * (1 + 2.0 ** -22 * np.arange(-6, 7))]).astype(np.float32)
    x = x[x != 1]
    lib = _native.load()
    with g.make(rule, one * big, one, one, eps=0.0, quality_interval=1) as job:
        dW, dH = _factors(job)

        def sample(h):
            dW.fill_(1.0)
            dH.fill_(float(h))
            torch.cuda.synchronize()
            _native.check(lib.gpunmf_factors_changed(job._h))
            job.DoIteration(False)
            job.Synchronize()

        for _ in range(4):  # the improvement is that of the two samples before
            sample(1.0)
        for v in x:
            sample(v)     # takes it
            sample(1.0)   # reads it, after one of W H = 1: -1
            want = float(big) * np.log10(float(v))
            assert abs(job.QualityImprovement() - want) <= 4 * 2.0 ** -23 * abs(want), float(v)


@pytest.mark.gpu
@pytest.mark.parametrize("eps", [1e-8, 1e-3])
def test_quotient(eps):
    rng = np.random.default_rng(1)
    m = 5000
    eps = np.float32(eps)
    V = (rng.random((1, m)) * 2.0 ** rng.uniform(-10, 10, (1, m))).astype(np.float32)
    H = (2.0 ** rng.integers(-12, 13, (1, m))).astype(np.float32)
    with g.make(1, V, np.ones((1, 1), dtype=np.float32), H, eps=float(eps), quality_interval=0) as job:
        job.DoIteration(False)
        got = job.GetH() / H
    want = V / (H + eps)
    assert np.max(np.abs(got.astype(np.float64) - want) / np.spacing(want)) <= 1.0
