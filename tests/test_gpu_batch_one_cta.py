"""Batches run by the one persistent launch, one CTA an instance: every rank class, V strides with n % 4 != 0, edges of
tiles and chunks, its graph's replays, its tile configurations, and the two ways to run a batch one after the
other.  Against FP64; its sums are FP32 multiply-adds of positive terms in chains of at most 1024: 1e-4 of a value
is 1600 roundings after one iteration."""
import numpy as np
import pytest

from gpumlib_gb300 import batch as gb
from gpumlib_gb300._native import GpuNmfError
from test_gpu_split_batch import EPS, _instance, _step64

TOL = 1e-4
SHAPES = [(64, 64, 4), (65, 33, 3), (130, 70, 8), (127, 100, 5), (90, 61, 16), (1, 7, 2), (61, 90, 13), (70, 75, 32), (35, 38, 27),
          (1021, 30, 9), (30, 509, 20)]


def _batch(shapes=SHAPES, seed=0):
    insts = [_instance(*s, seed=seed + k) for k, s in enumerate(shapes)]
    b = gb.Batch(insts, eps=EPS)
    b.share_launches(False)
    assert not b.shares_launches
    return insts, b


def _check(d, got, steps):
    V, W, H = (d[x].astype(np.float64) for x in "VWH")
    for _ in range(steps):
        W, H = _step64(V, W, H)
    assert np.max(np.abs(got[1] - H) / H) <= steps * TOL and np.max(np.abs(got[0] - W) / W) <= 2 * steps * TOL


@pytest.mark.gpu
def test_which_way():
    """Few and small: one launch; uneven and large: shared ones."""
    with gb.Batch([_instance(64, 64, 4, 0)]) as b:
        assert not b.shares_launches
        with pytest.raises(GpuNmfError):
            b.share_launches(True)
    with gb.Batch([_instance(128, 100, 8, k) for k in range(400)], eps=EPS) as b:
        assert not b.shares_launches
        b.run(1)
        _check(_instance(128, 100, 8, 399), b.get(399), 1)
    with gb.Batch([_instance(600, 400, 16, k) for k in range(20)]) as b:
        assert b.shares_launches


@pytest.mark.gpu
def test_against_fp64():
    insts, b = _batch()
    with b:
        b.run(1)
        for k, d in enumerate(insts):
            _check(d, b.get(k), 1)
        res = b.residuals()
        for k, d in enumerate(insts):
            W, H = b.get(k)
            want = np.linalg.norm(d["V"] - W.astype(np.float64) @ H) / np.linalg.norm(d["V"].astype(np.float64))
            assert abs(res[k] - want) <= 1e-6


@pytest.mark.gpu
def test_configurations_agree():
    insts, b = _batch(seed=50)
    ranks = gb.configs()
    with b:
        seen = 0
        for c, rc in enumerate(ranks):
            members = [k for k, s in enumerate(SHAPES) if gb.rank_class(s[2]) == rc]
            for k in members:
                b.set_config(k, c)
            b.commit()
            b.reset_factors()
            b.run(2)
            for k in members:
                _check(insts[k], b.get(k), 2)
                seen += 1
        assert seen >= len(ranks)


@pytest.mark.gpu
def test_replays_continue():
    _, a = _batch(seed=70)
    _, b = _batch(seed=70)
    with a, b:
        for _ in range(3):
            a.run(4)
        b.run(12)
        for k in range(a.count):
            assert all(np.array_equal(x, y) for x, y in zip(a.get(k), b.get(k)))


@pytest.mark.gpu
def test_one_way_and_the_other():
    shapes = [(600, 400, 16), (257, 129, 32), (130, 500, 10), (333, 222, 4)] * 6
    insts = [_instance(*s, seed=k) for k, s in enumerate(shapes)]
    with gb.Batch(insts, eps=EPS) as b:
        assert b.shares_launches
        b.run(1)
        b.share_launches(False)
        b.run(1)
        b.share_launches(True)
        b.run(1)
        for k in range(4):
            _check(insts[k], b.get(k), 3)


@pytest.mark.gpu
def test_autotune_of_a_batch_that_runs_this_way():
    insts = [_instance(128, 100, 8, k) for k in range(300)]
    with gb.Batch(insts) as b:
        assert not b.shares_launches
        table = gb.autotune(b, insts, sample=60, iters=2)
        assert all(len(timings) == sum(rc == key[0] for rc in gb.configs()) for key, (_, timings) in table.items())
        assert len(set(b.cfg)) == 1
        b.run(2)
        _check(insts[5], b.get(5), 2)
