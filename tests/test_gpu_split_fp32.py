"""FP32 jobs of rank <= 128 (products on the tensor cores as six BF16 products of three-part operands):
one iteration against FP64 at the edges of its tiles (128 rows), chunks (64 of K), rank classes
(32 / 64 / 128) and V strides (n % 4), the residual, and infinities and NaN.

Tolerance: V, W and H are positive, so every sum's relative error is at most that of its terms plus
its additions'.  Dropped products of parts: 2^-23.  An accumulator takes 24 additions that may
truncate (2^-23 each; the five small products' ones weigh 2^-8): 4 * 2^-23 + 20 * 2^-31.  The chunk sums:
at most K / 64 + slots <= 72 roundings of 2^-24 here.  The Gram and denominator sums: at most 2100
roundings in chains of <= 128, and the update four more.  Together below 256 * 2^-24 = 1.6e-5."""
import numpy as np
import pytest

import gpumlib_gb300 as g

TOL = 1.6e-5
EPS = 1e-8


def _inputs(n, m, r, seed):
    rng = np.random.default_rng(seed)
    return (rng.random((n, m), dtype=np.float32) + np.float32(0.01), rng.random((n, r), dtype=np.float32) + np.float32(0.01),
            rng.random((r, m), dtype=np.float32) + np.float32(0.01))


def _step64(rule, V, W, H):
    V, W, H = (x.astype(np.float64) for x in (V, W, H))
    if rule == 0:
        H = H * ((W.T @ V) / (W.T @ W @ H + EPS))
        return W * ((V @ H.T) / (W @ (H @ H.T) + EPS)), H
    H = H * ((W.T @ (V / (W @ H + EPS))) / W.sum(0)[:, None])
    return W * (((V / (W @ H + EPS)) @ H.T) / H.sum(1)[None, :]), H


SHAPES = [(1, 1, 1), (127, 129, 16), (128, 64, 17), (129, 65, 32), (130, 191, 33), (63, 1000, 64), (1000, 61, 65),
          (257, 385, 112), (512, 640, 128), (2049, 515, 48), (4096, 300, 97)]


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("n,m,r", SHAPES)
def test_one_iteration(rule, n, m, r):
    V, W, H = _inputs(n, m, r, n + m + r)
    with g.make(rule, V, W, H, eps=EPS) as job:
        job.DoIteration()
        Wg, Hg, res = job.GetW(), job.GetH(), job.Residual()
    We, He = _step64(rule, V, W, H)
    assert np.max(np.abs(Hg - He) / He) <= TOL
    assert np.max(np.abs(Wg - We) / We) <= 2 * TOL  # from an H that is TOL off
    exact = np.linalg.norm(V - Wg.astype(np.float64) @ Hg) / np.linalg.norm(V.astype(np.float64))
    assert abs(res - exact) <= 1e-6 * max(1.0, exact)  # V - W H, W H within 64 * 2^-24 of its value


@pytest.mark.gpu
def test_same_bits_every_time():
    # zero entries and a many-chunk stream (a V stage must not be refilled before it is read)
    rng = np.random.default_rng(3)
    n, m, r = 4096, 2048, 128
    V = rng.poisson(2.0, (n, m)).astype(np.float32)
    _, W, H = _inputs(n, m, r, 4)
    got = []
    for _ in range(4):
        with g.make(1, V, W, H, eps=EPS) as job:
            job.Iterate(2)
            got.append((job.GetW(), job.GetH()))
    assert all(np.array_equal(w, got[0][0]) and np.array_equal(h, got[0][1]) for w, h in got)


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_infinity_and_nan_in_v(rule, bad):
    V, W, H = _inputs(150, 200, 20, 7)
    W[::3] = 0.5  # exact in one part: its other parts are zero
    V[7, 9] = bad
    with g.make(rule, V, W, H, eps=EPS) as job:
        job.DoIteration(False)
        Hg = job.GetH()
    clean = np.delete(Hg, 9, axis=1)
    assert np.isfinite(clean).all()
    if np.isnan(bad):
        assert np.isnan(Hg[:, 9]).all()
    elif rule == 0:
        assert np.isposinf(Hg[:, 9]).all()  # formed again by plain FP32 sums
    else:
        assert not np.isfinite(Hg[:, 9]).any()


def test_three_parts_hold_a_float():
    """The cut, restated: the nearest BF16 of what is left, three times, is exact for every normal float
    well above the smallest, and the six products of parts are a product to 2^-23 (2 * 2^-8 * 2^-16, and 2^-32)."""
    rng = np.random.default_rng(0)

    def cut(x):
        def near(v):  # to 8 significand bits, ties to even
            u = v.view(np.uint32)
            return ((u + np.uint32(0x7FFF) + ((u >> np.uint32(16)) & np.uint32(1))) & np.uint32(0xFFFF0000)).view(np.float32)
        a = near(x)
        b = near(x - a)
        return a, b, (x - a) - b

    x = (rng.random(200000, dtype=np.float32) * np.exp2(rng.integers(-90, 90, 200000))).astype(np.float32)
    y = (rng.random(200000, dtype=np.float32) + np.float32(1e-3)).astype(np.float32)
    p, q = cut(x), cut(y)
    for parts, v in ((p, x), (q, y)):
        assert np.array_equal(sum(z.astype(np.float64) for z in parts), v.astype(np.float64))
        assert all(np.array_equal(z.view(np.uint32) & 0xFFFF, np.zeros(z.size, np.uint32)) for z in parts)
    six = sum(p[i].astype(np.float64) * q[j] for i in range(3) for j in range(3 - i))
    exact = x.astype(np.float64) * y
    assert np.max(np.abs(six - exact) / np.where(exact > 0, exact, 1)) <= 2.0 ** -23 * (1 + 2.0 ** -7)
