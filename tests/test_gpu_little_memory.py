"""An FP32 job for which there is memory on the CUDA cores but not on the tensor cores (V a second time, with
padded columns): it is made all the same.  One iteration against FP64 (bound: test_gpu_split_fp32)."""
import numpy as np
import pytest
import torch

import gpumlib_gb300 as g
from gpumlib_gb300 import _native
from test_gpu_split_fp32 import EPS, TOL, _inputs, _step64

N, M, R = 5001, 20000, 3  # 400 MB of V; columns of 5001 want padding


@pytest.mark.gpu
def test_job_without_room_for_the_padded_copy():
    lib = _native.load()
    V, W, H = _inputs(N, M, R, 0)
    V = np.asfortranarray(V)
    small = _inputs(130, 70, R, 1)
    for r in (R, 140):  # the kernels of both paths are loaded while there is memory
        with g.make(0, small[0], np.tile(small[1], (1, 50))[:, :r], np.tile(small[2], (50, 1))[:r]) as job:
            job.DoIteration()
            job.Residual()
    _native.check(lib.gpunmf_trim_pool())
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    taken = torch.empty(free - 700 * 1024 * 1024, dtype=torch.uint8, device="cuda")  # 700 MB left: V once and its workspaces
    try:
        with g.make(0, V, W, H, eps=EPS, quality_interval=0) as job:
            job.DoIteration()
            Wg, Hg, res = job.GetW(), job.GetH(), job.Residual()
        _native.check(lib.gpunmf_trim_pool())
    finally:
        del taken
        torch.cuda.empty_cache()
    We, He = _step64(0, V, W, H)
    assert np.max(np.abs(Hg - He) / He) <= TOL and np.max(np.abs(Wg - We) / We) <= 2 * TOL
    want = np.linalg.norm(V - Wg.astype(np.float64) @ Hg) / np.linalg.norm(V.astype(np.float64))
    assert abs(res - want) <= 1e-6
