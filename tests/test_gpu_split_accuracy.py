"""How near FP64 the FP32 products are: the drift of the factors over many iterations, and every one of the
six products of parts.

Drift.  The scale between W(:, a) and H(a, :) is free, so a numerator that is off by the same fraction in
every iteration adds up.  Rounding to nearest leaves the mean of a factor's relative errors within 2^-24 / sqrt(entries)
an iteration, well below 1e-9 of it here; what the tensor cores' cut leaves, after the correction for
it, is at most a fifth of 2^-24 apart between the two half-steps (its measured spread over data, sp_low_sum).
100 iterations: 100 * 0.2 * 2^-24 = 1.2e-6 of the mean signed error.

Parts.  x = 1 + 2^-8 + 2^-8 (2^-8 + 2^-9) and like values have second and third parts of one sign and near their largest
(2^-8 and 2^-17 of x), so a product that is missing moves the sum by 2^-17 = 7.6e-6 of it, or more.  The sum itself, of 16 terms
in one chunk, is 24 additions cut at 2^-23 and fewer than ten roundings of 2^-24 beside them (the Gram and
denominator sums of 16 terms: 32 more at most): below 3e-6."""
import numpy as np
import pytest

import gpumlib_gb300 as g
from gpumlib_gb300.batch import Batch

EPS = 1e-8


def _u(rng, *s):
    return rng.random(s, dtype=np.float32) + np.float32(0.01)


def _steps64(rule, V, W, H, iters):
    V, W, H = (x.astype(np.float64) for x in (V, W, H))
    for _ in range(iters):
        if rule == 0:
            H = H * ((W.T @ V) / (W.T @ W @ H + EPS))
            W = W * ((V @ H.T) / (W @ (H @ H.T) + EPS))
        else:
            H = H * ((W.T @ (V / (W @ H + EPS))) / W.sum(0)[:, None])
            W = W * (((V / (W @ H + EPS)) @ H.T) / H.sum(1)[None, :])
    return W, H


def _means(got, want):
    return max(abs(float(np.mean((a.astype(np.float64) - b) / b))) for a, b in zip(got, want))


# K of the H-step (n) and of the W-step (m): 1, 2, 3 and 32 chunks of 64, full and with a remainder of 1 .. 4 steps
SIDES = [(64, 2048), (2048, 64), (70, 300), (300, 70), (100, 2048), (2048, 113), (128, 64), (192, 700), (65, 2040), (512, 512)]


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("n,m", SIDES)
def test_no_drift(rule, n, m):
    rng = np.random.default_rng(n * 7 + m)
    r = 20
    V, W, H = _u(rng, n, 6) @ _u(rng, 6, m) + _u(rng, n, m), _u(rng, n, r), _u(rng, r, m)
    with g.make(rule, V, W, H, eps=EPS, quality_interval=0) as job:
        job.Iterate(100)
        got = job.GetW(), job.GetH()
    assert _means(got, _steps64(rule, V, W, H, 100)) <= 1.2e-6


@pytest.mark.gpu
def test_no_drift_in_batches():
    rng = np.random.default_rng(1)
    insts = [{"V": _u(rng, n, m), "W": _u(rng, n, 14), "H": _u(rng, 14, m)} for n, m in SIDES if max(n, m) <= 700] * 3
    with Batch(insts, eps=EPS) as b:
        b.run(100)
        b.synchronize()
        for k, d in enumerate(insts[:len(insts) // 3]):
            assert _means(b.get(k), _steps64(0, d["V"], d["W"], d["H"], 100)) <= 1.2e-6


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("r", [3, 40, 100])
def test_every_product_of_parts_counts(rule, r):
    n, m = 16, 300
    rng = np.random.default_rng(r)

    def parts(*s):  # 1 + second part + third part, both near their largest and above zero
        x = np.float64(1) + 2.0 ** -8 * (1 - 2.0 ** -7 * rng.integers(1, 8, s)) + 2.0 ** -17 * (1 - 2.0 ** -6 * rng.integers(1, 4, s))
        return x.astype(np.float32)

    V, W, H = parts(n, m), parts(n, r), parts(r, m)
    with g.make(rule, V, W, H, eps=EPS, quality_interval=0) as job:
        job.Iterate(1, False)
        Hg = job.GetH()
    V, W, H = (x.astype(np.float64) for x in (V, W, H))
    if rule == 0:
        want = H * ((W.T @ V) / (W.T @ W @ H + EPS))
    else:
        want = H * ((W.T @ (V / (W @ H + EPS))) / W.sum(0)[:, None])
    assert np.max(np.abs(Hg - want) / want) <= 3e-6
