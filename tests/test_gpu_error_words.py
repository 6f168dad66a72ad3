"""A wait that ran out is reported by every call that hands results out: jobs, batches, the server.  The error word
is set from the host as a kernel that gave up sets it (no kernel is made to fail); what comes after is whole."""
import threading

import numpy as np
import pytest

import gpumlib_gb300 as g
from gpumlib_gb300 import _native
from gpumlib_gb300.batch import Batch
from gpumlib_gb300.serve import Server
from test_gpu_split_batch import EPS, TOL, _instance, _step64

TIMEOUT, UNSUPPORTED = 6, 4


def _status(call):
    with pytest.raises(g.GpuNmfError) as e:
        call()
    assert "gave up waiting" in str(e.value)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("rule", [0, 1])
def test_job(rule, precision):
    d = _instance(300, 200, 20, 1)
    lib = _native.load()
    with g.make(rule, d["V"], d["W"], d["H"], precision=precision) as job:
        job.Iterate(2)
        _native.check(lib.gpunmf_inject_error_word(job._h))
        for call in (job.Synchronize, job.GetW, job.GetH, job.GetWH, job.Residual, job.ObjectiveKL):
            _status(call)
    with g.make(rule, d["V"], d["W"], d["H"], precision=precision) as job:
        job.Iterate(2)
        assert np.isfinite(job.Residual())


@pytest.mark.gpu
def test_job_without_waits():
    d = _instance(200, 180, 140, 1)
    with g.make(0, d["V"], d["W"], d["H"]) as job:
        assert _native.load().gpunmf_inject_error_word(job._h) == UNSUPPORTED


@pytest.mark.gpu
def test_batch():
    insts = [_instance(300, 200, 8, k) for k in range(20)]
    lib = _native.load()
    with Batch(insts, eps=EPS) as b:
        b.run(1)
        _native.check(lib.gpunmf_batch_inject_error_word(b._h))
        for call in (lambda: b.get(0), lambda: b.get(1), b.residuals, lambda: b.time(1), b.synchronize):
            _status(call)
        b.reset_factors()
        b.run(1)
        W, H = b.get(7)
        b.synchronize()
    W1, H1 = _step64(*(insts[7][x].astype(np.float64) for x in "VWH"))
    assert np.max(np.abs(H - H1) / H1) <= TOL and np.max(np.abs(W - W1) / W1) <= 2 * TOL


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_server(precision):
    with Server(slots=2, precision=precision, tol=0.0, max_iters=30) as server:
        _native.check(_native.load().gpunmf_server_inject_error_word(server._h))
        for k in range(4):
            server.submit(k, k % 2, 300, 260, 20, seed=k)
        assert server.drain(60.0)
        status = [r["status"] for r in server.poll()]
    assert sorted(status) == [0, 0, 0, TIMEOUT]


@pytest.mark.gpu
def test_two_threads_read_a_batch():
    insts = [_instance(900 - 3 * k, 200 + k, 8, k) for k in range(40)]
    with Batch(insts, eps=EPS) as b:
        b.run(2)
        want = [b.get(k) for k in range(b.count)]
        wrong = []

        def read(first):
            for _ in range(20):
                for k in range(first, b.count, 2):
                    w, h = b.get(k)
                    if not (np.array_equal(w, want[k][0]) and np.array_equal(h, want[k][1])):
                        wrong.append(k)

        threads = [threading.Thread(target=read, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not wrong
