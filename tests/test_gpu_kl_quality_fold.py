"""KL jobs sample the quality inside their H-step: the lagged improvement against FP64, at the edges of the
tiles (128 rows), of the K blocks (128 in BF16, 64 in FP32) and of the rank classes.

The expected sums are of each iteration's own factors (from a second job that does not sample: the sample
changes no factor, so both agree bit for bit), rounded as the precision rounds them.  Tolerance, per unit of
sum |V log10(S + eps)| + V + S: S, at most 128 truncating additions of 2^-23; the logarithm moves by that
over ln 10, and its own error is 2^-21 of a bit; the running sums take at most 256 roundings of 2^-24; the
word read back is rounded to 2^-24.  Together below 5e-5, twice that for a difference of two samples."""
import numpy as np
import pytest

import gpumlib_gb300 as g

EPS = 1e-6


def _bf16(x):
    u = np.ascontiguousarray(x, dtype=np.float32).view(np.uint32)
    u = (u + np.uint32(0x7FFF) + ((u >> np.uint32(16)) & np.uint32(1))) & np.uint32(0xFFFF0000)
    return u.view(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("rule", [1, 3])
@pytest.mark.parametrize("n,m,r", [(1, 1, 1), (127, 129, 16), (129, 257, 17), (300, 515, 64), (515, 300, 65), (640, 2049, 128)])
def test_folded_sample(precision, rule, n, m, r):
    rng = np.random.default_rng(n + m + r)
    V = np.asfortranarray(rng.poisson(3.0, (n, m)).astype(np.float32)) + np.float32(1)  # exact in BF16
    W = np.asfortranarray(rng.random((n, r), dtype=np.float32) + np.float32(0.05))
    H = np.asfortranarray(rng.random((r, m), dtype=np.float32) + np.float32(0.05))
    values, sizes, got = [], [], []
    with g.make(rule, V, W, H, eps=EPS, precision=precision, quality_interval=1) as job, \
            g.make(rule, V, W, H, eps=EPS, precision=precision, quality_interval=0) as plain:
        for _ in range(5):
            w, h = plain.GetW(), plain.GetH()
            if precision == "bf16":
                w, h = _bf16(w), _bf16(h)
            S = w.astype(np.float64) @ h.astype(np.float64)
            L = V * np.log10(S + EPS)
            values.append((L - S).sum())
            sizes.append(np.abs(L).sum() + V.sum() + S.sum())
            job.DoIteration()
            plain.DoIteration()
            got.append(job.QualityImprovement())
        assert np.array_equal(job.GetW(), plain.GetW()) and np.array_equal(job.GetH(), plain.GetH())
    # a sample reads the previous iteration's value, and the first two leave the improvement at 1
    assert got[0] == got[1] == 1.0
    for k in range(2, 5):
        assert abs(got[k] - (values[k - 1] - values[k - 2])) <= 1e-4 * max(sizes[k - 2:k])
