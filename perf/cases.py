"""What this framework is asked to do in earnest, as cases that can be timed.

Every case goes through the public entry points: the NMF classes of ``gpumlib_gb300`` (the mirror of
the C++ classes), ``batch.Batch`` and ``serve.Server``.  A pass of an ``iterate`` or ``monitor`` case
leaves its results in the job's own device factors (``gpunmf_device_factors``), as a program that keeps
iterating does; ``train``, ``factorize``, ``batch`` and ``serving`` read them back to the host, as
programs at their end do.

Sizes are those of the repository's benchmark workloads (1024 x 512 r = 16, 8192 x 8192 r = 64,
16384 x 4096 r = 128 counts, uneven batches, the serving stream), of the face data set its tests use
(361 x 2429, rank 49, and its 472 test images), and generic odd ones.
"""
import ctypes
import math
import random

import numpy as np
import torch

from gpumlib_gb300 import _native, nmf as _nmf
from gpumlib_gb300.batch import Batch
from gpumlib_gb300.serve import Server

REFERENCE_EPS = float(np.float32(1e-8))
SERVING_EPS = float(np.float32(1e-9))


def _job(name, kind, rule, n, m, r, precision, iters, quality=1, data="lowrank", update_w=True):
    return {"name": name, "kind": kind, "rule": rule, "n": n, "m": m, "r": r, "precision": precision,
            "iters": iters, "quality": quality, "data": data, "update_w": update_w}


def listed():
    return [
        # one DoIteration of a small plain job with the default quality sampling: the smallest call
        _job("plain_small", "iterate", 0, 1024, 512, 16, "fp32", 1, data="uniform"),
        # FacesNMF's training loop: DoIteration and QualityImprovement until done, then GetW / GetH
        _job("faces_train", "train", 0, 361, 2429, 49, "fp32", 20, data="faces"),
        # the codes of the face test set under a trained W: H steps only (DoIteration(false))
        _job("faces_encode_kl", "iterate", 1, 361, 472, 49, "fp32", 10, quality=0, data="faces", update_w=False),
        # the large plain job, as the class runs it by default (quality sampled every iteration)
        _job("euclid_fp32", "iterate", 0, 8192, 8192, 64, "fp32", 2),
        # the plain KL job on counts, default quality sampling
        _job("kl_fp32", "iterate", 1, 16384, 4096, 128, "fp32", 1, data="counts"),
        # the additive KL rule on an odd shape
        _job("additive_kl_fp32", "iterate", 3, 3001, 1777, 40, "fp32", 4, quality=0),
        # the headline: a run of iterations of the large job in BF16
        _job("euclid_bf16", "iterate", 0, 8192, 8192, 64, "bf16", 20, quality=0),
        # a rank over 64, checked for convergence every ten iterations (FP64 residual), as the server does
        _job("monitored_bf16", "monitor", 0, 5000, 3001, 100, "bf16", 10, quality=0),
        # KL on counts in BF16, default quality sampling
        _job("kl_bf16", "iterate", 1, 16384, 4096, 128, "bf16", 10, data="counts"),
        # a whole factorisation from host matrices to host factors
        _job("factorize_bf16", "factorize", 0, 4096, 2048, 32, "bf16", 50),
        # hundreds of uneven small factorisations in one launch, all factors read back
        {"name": "batch_uneven", "kind": "batch", "count": 768, "iters": 50, "shapes": 1},
        # a burst of jobs through the server: generated on the device, admitted, iterated, fetched
        {"name": "serving_burst", "kind": "serving", "jobs": 24, "iters": 100, "shapes": 1, "precision": "bf16"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["iterate"] * 7 + ["train", "monitor", "monitor", "factorize", "batch", "serving"])
    if kind == "batch":
        return {"kind": kind, "count": _log_uniform(rng, 48, 768), "iters": rng.randint(5, 50),
                "shapes": rng.randrange(1 << 20)}
    if kind == "serving":
        return {"kind": kind, "jobs": rng.randint(4, 24), "iters": rng.randint(2, 10) * 10,
                "shapes": rng.randrange(1 << 20), "precision": rng.choice(["bf16", "bf16", "fp32"])}
    precision = rng.choice(["fp32", "bf16"])
    rule = rng.choice([0, 0, 0, 1, 1, 2, 3, 4])
    top = 2048 if kind in ("train", "factorize") else 8192
    n, m = _log_uniform(rng, 64, top), _log_uniform(rng, 64, top)
    r = min(_log_uniform(rng, 2, 128), n, m)
    c = _job("", kind, rule, n, m, r, precision, rng.choice([1, 2, 5, 10]))
    del c["name"]
    c["quality"] = rng.choice([1, 1, 0]) if kind != "monitor" else 0
    c["data"] = rng.choice(["counts", "sparse"]) if rule == 1 else rng.choice(["lowrank", "uniform"])
    c["update_w"] = rng.random() < 0.85 or rule == 4  # rule 4 has no H step
    return c


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _matrices(case, seed):
    """V' (m x n), W' (r x n), H' (m x r) in FP32 on the GPU: the transposes, so that their rows are
    the columns that the framework's column-major matrices hold."""
    g = _gen(seed)
    n, m, r = case["n"], case["m"], case["r"]
    data = case["data"]
    if data == "uniform":
        V = _uniform(g, m, n) + 1e-3
    elif data in ("counts", "sparse"):
        # counts with a low-rank mean of skewed weights; sparse: about nine zeros in ten
        P = -torch.log1p(-_uniform(g, r, n)) * _uniform(g, r, n) ** 3
        Q = -torch.log1p(-_uniform(g, m, r)) * _uniform(g, m, r) ** 3
        lam = Q @ P
        lam *= (8.0 if data == "counts" else 0.12) / lam.mean()
        V = torch.poisson(lam, generator=g)
        del lam
    else:
        # low rank, Gamma(2, 0.5) factors, and a little positive noise
        A = -0.5 * (torch.log1p(-_uniform(g, r, n)) + torch.log1p(-_uniform(g, r, n)))
        B = -0.5 * (torch.log1p(-_uniform(g, m, r)) + torch.log1p(-_uniform(g, m, r)))
        V = B @ A
        if data == "faces":  # grey levels of 8 bits, scaled to [0, 1]
            V = torch.round(255.0 * (V / V.max()).sqrt()) / 255.0
        else:
            V += 0.01 * torch.randn(m, n, generator=g, device="cuda").abs()
    W = _uniform(g, r, n) + 1e-4
    H = _uniform(g, m, r) + 1e-4
    return V, W, H


def _host(t):
    return t.cpu().numpy().T  # column-major, no further copy


def _uneven(case):
    """The (n, m, r) of a batch: as its workload draws them."""
    rng = random.Random(case["shapes"])
    return [(rng.randint(32, 1024), rng.randint(32, 512), rng.choice((4, 8, 16, 32))) for _ in range(case["count"])]


def _stream_jobs(case):
    """(rule, n, m, r) of a burst of served jobs."""
    rng = random.Random(case["shapes"])
    return [(1 if rng.random() < 0.3 else 0, _log_uniform(rng, 64, 2048), _log_uniform(rng, 64, 2048), rng.randint(8, 64))
            for _ in range(case["jobs"])]


def _instances(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for n, m, r in _uneven(case):
        draw01 = lambda a, b: rng.random((b, a), dtype=np.float32).T  # noqa: E731
        out.append({"V": draw01(n, m), "W": draw01(n, r) + np.float32(1e-4), "H": draw01(r, m) + np.float32(1e-4)})
    return out


class _DeviceMatrix:
    """A job's device factor under the CUDA array interface (rows are the matrix's columns); it
    keeps the job, whose memory it is."""

    def __init__(self, job, ptr, shape):
        self.job = job
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}


def _device_factors(job):
    w, h = ctypes.c_void_p(), ctypes.c_void_p()
    _native.check(_native.load().gpunmf_device_factors(job._h, ctypes.byref(w), ctypes.byref(h)))
    return {"W": torch.as_tensor(_DeviceMatrix(job, w.value, (job.r, job.n)), device="cuda"),
            "H": torch.as_tensor(_DeviceMatrix(job, h.value, (job.m, job.r)), device="cuda")}


def prepare(case, seed):
    state = {"case": case}
    if case["kind"] == "batch":
        state["batch"] = Batch(_instances(case, seed))
        return state
    if case["kind"] == "serving":
        state["seeds"] = [1000 * int(seed) + i for i in range(case["jobs"])]
        state["jobs"] = _stream_jobs(case)
        return state
    V, W, H = (_host(t) for t in _matrices(case, seed))
    if case["kind"] == "factorize":
        state["host"] = (V, W, H)
        return state
    job = _nmf.make(case["rule"], V, W, H, precision=case["precision"], quality_interval=case["quality"])
    state["job"] = job
    state["factors"] = _device_factors(job)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "iterate":
        state["job"].Iterate(case["iters"], case["update_w"])
        return state["factors"]
    if kind == "monitor":
        state["job"].Iterate(case["iters"], case["update_w"])
        return dict(state["factors"], residual=state["job"].Residual())
    if kind == "train":
        job = state["job"]
        for _ in range(case["iters"]):
            job.DoIteration(case["update_w"])
            if job.QualityImprovement() < -1e30:  # the loop's stop test, at a tolerance it does not reach
                break
        return {"W": job.GetW(), "H": job.GetH()}
    if kind == "factorize":
        with _nmf.make(case["rule"], *state["host"], precision=case["precision"], quality_interval=case["quality"]) as job:
            for _ in range(case["iters"]):
                job.DoIteration(case["update_w"])
            return {"W": job.GetW(), "H": job.GetH()}
    if kind == "batch":
        batch = state["batch"]
        batch.run(case["iters"])
        got = [batch.get(k) for k in range(batch.count)]
        return {"W": np.concatenate([w.ravel(order="K") for w, _ in got]),
                "H": np.concatenate([h.ravel(order="K") for _, h in got])}
    with Server(slots=16, precision=case["precision"], tol=1e-3, max_iters=case["iters"], keep_factors=True) as server:
        for k, (rule, n, m, r) in enumerate(state["jobs"]):
            server.submit(k, rule, n, m, r, state["seeds"][k])
        server.drain(60.0)
        out = {}
        for k, (_, n, m, r) in enumerate(state["jobs"]):
            _, out["W%d" % k], out["H%d" % k] = server.fetch(k, n, m, r)
        return out


# ------------------------------------------------------------------ the work

def _iteration(rule, n, m, r, element, update_w):
    """Bytes and operations of one iteration: each half-step reads V once (its factor depends on all of
    the other one's), reads the other factor and reads and writes its own."""
    halves = (rule != 4) + bool(update_w)
    kl = rule in (1, 3)
    flops = halves * (4.0 if kl else 2.0) * n * m * r
    if not kl:
        flops += 4.0 * r * r * (n + m) * halves / 2.0
    return halves * (element * n * m + 6.0 * (n + m) * r), flops


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for n, m, r in _uneven(case):
            b += 4.0 * (n * m + 2 * (n + m) * r)  # an instance's V fits on chip: once for all iterations
            f += case["iters"] * _iteration(0, n, m, r, 4.0, True)[1]
        return {"bytes": b, "flops": f}
    element = 2.0 if case["precision"] == "bf16" else 4.0
    if kind == "serving":
        b = f = 0.0
        for rule, n, m, r in _stream_jobs(case):
            bi, fi = _iteration(rule, n, m, r, element, True)
            # V is made once, and a residual is formed after every ten iterations
            b += case["iters"] * bi + 4.0 * n * m + case["iters"] / 10 * 4.0 * n * m
            f += case["iters"] * fi + case["iters"] / 10 * 2.0 * n * m * r + 2.0 * n * m * r
        return {"bytes": b, "flops": f}
    n, m, r = case["n"], case["m"], case["r"]
    b, f = _iteration(case["rule"], n, m, r, element, case["update_w"])
    if case["quality"]:  # a sample needs W H, and V beside the half-steps' passes can be shared
        f += 2.0 * n * m * r
    b, f = case["iters"] * b, case["iters"] * f
    if kind == "monitor":
        b, f = b + 4.0 * n * m, f + 2.0 * n * m * r
    if kind == "factorize":
        b += 4.0 * (n * m + 2 * (n + m) * r)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ the same in 64 bits

def _step(rule, V, W, H, eps, update_w):
    """One iteration of a rule in FP64, on matrices of the usual shapes (W n x r, H r x m)."""
    if rule in (0, 2, 4):
        if rule != 4:
            num, den = W.T @ V, (W.T @ W) @ H
            H = H * (num / (den + eps)) if rule == 0 else torch.clamp(H + H / den * (num - den), min=0)
        if update_w:
            num, den = V @ H.T, W @ (H @ H.T)
            W = W * (num / (den + eps)) if rule == 0 else torch.clamp(W + W / den * (num - den), min=0)
        return W, H
    less = 1.0 if rule == 3 else 0.0
    R = V / (W @ H + eps) - less
    s = torch.clamp(W.sum(0), min=eps)[:, None]
    H = H * ((W.T @ R) / s) if rule == 1 else torch.clamp(H + H / s * (W.T @ R), min=0)
    if update_w:
        R = V / (W @ H + eps) - less
        s = torch.clamp(H.sum(1), min=eps)[None, :]
        W = W * ((R @ H.T) / s) if rule == 1 else torch.clamp(W + W / s * (R @ H.T), min=0)
    return W, H


def _uniform_counters(seed, stream, count):
    """The served jobs' counter generator: splitmix64 of (key + (k + 1) golden), its top 24 bits."""
    with np.errstate(over="ignore"):
        key = np.uint64(((int(seed) * 0xD1B54A32D192ED03 + 0x8CB92BA72F3D8DD7) & (2**64 - 1)) ^ (stream << 56))
        z = key + np.arange(1, count + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    return (z >> np.uint64(40)).astype(np.float32) * np.float32(1.0 / 16777216.0)


def _served_inputs(n, m, r, seed):
    """V, W, H of a served job: V = A B + |N(0, 0.01)| by Box-Muller, A, B, W, H uniform."""
    mat = lambda x, rows, cols: torch.from_numpy(x.reshape(cols, rows)).cuda().double().T  # noqa: E731
    A, B = mat(_uniform_counters(seed, 0, n * r), n, r), mat(_uniform_counters(seed, 1, r * m), r, m)
    u = torch.from_numpy(_uniform_counters(seed, 2, 2 * n * m)).cuda().double()
    z = torch.sqrt(-2.0 * torch.log(u[0::2] + 0.5 / 16777216.0)) * torch.cos(2.0 * math.pi * u[1::2])
    V = ((A @ B).float() + (0.01 * z).abs().float().reshape(m, n).T).double()
    W = mat(_uniform_counters(seed, 3, n * r) + np.float32(1e-4), n, r)
    H = mat(_uniform_counters(seed, 4, r * m) + np.float32(1e-4), r, m)
    return V, W, H


def _flat(t):
    return t.T.contiguous()  # the framework's column-major order


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        Ws, Hs = [], []
        for d in _instances(case, seed):
            V, W, H = (torch.from_numpy(np.ascontiguousarray(d[k])).cuda().double() for k in "VWH")
            for _ in range(case["iters"]):
                W, H = _step(0, V, W, H, REFERENCE_EPS, True)
            Ws.append(_flat(W).reshape(-1))
            Hs.append(_flat(H).reshape(-1))
        return {"W": torch.cat(Ws), "H": torch.cat(Hs)}
    if kind == "serving":
        out = {}
        for k, (rule, n, m, r) in enumerate(_stream_jobs(case)):
            V, W, H = _served_inputs(n, m, r, 1000 * int(seed) + k)
            for _ in range(case["iters"]):
                W, H = _step(rule, V, W, H, SERVING_EPS, True)
            out["W%d" % k], out["H%d" % k] = W.cpu().numpy(), H.cpu().numpy()
        return out
    V, W, H = (t.double().T for t in _matrices(case, seed))
    for _ in range(case["iters"]):
        W, H = _step(case["rule"], V, W, H, REFERENCE_EPS, case["update_w"])
    if kind in ("train", "factorize"):
        return {"W": W.cpu().numpy(), "H": H.cpu().numpy()}
    out = {"W": _flat(W), "H": _flat(H)}
    if kind == "monitor":
        out["residual"] = float(torch.linalg.norm(V - W @ H) / torch.linalg.norm(V))
    return out
