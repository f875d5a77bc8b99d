"""The work this library does for its users, as a list of timed cases.

Every case is one call (or the short fixed sequence of calls) that a program
makes through the public entry points, over the range of sizes, dimensions,
list lengths, bucket bounds and forms the library is used with: point sets of
a thousand to two million points, d in {64, 100, 128}, k from 10 to 100,
device-resident and host buffers, the 2-means and the KD splitter, FP32 and
BF16 estimates, single, batched and served builds, and the bucket pass on the
caller's own partition.

`listed()` names the cases, `draw()` gives further ones of the same ranges,
`prepare()` makes what a program holds before the call (points on the device
or the host, output buffers, a context or a server), `run()` makes the call,
`work()` counts what the path cannot do without, and `exact()` gives the 64-bit
result where the result is defined without this library's own choices (a set
that is one bucket, or the bucket pass on a given partition).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from sigmod23ann_b200 import KnngContext, KnngServer, Stats, default_params, kd_params, load_library

GIB = 1 << 30
# Device memory a context may hold: a third of the card and less, so that a
# program can keep several of them.
CONTEXT_BUDGET = 40 * GIB
SERVER_BUDGET = 44 * GIB


# --------------------------------------------------------------------- cases

def listed() -> list[dict]:
    return [
        # The smallest call: one set of a batch's smallest size, buckets of up
        # to 1,024 points, so that the whole set is a single bucket.
        dict(name="set-1k", form="device", n=1000, d=64, k=50, data="mixture16", max_leaf=1025, max_leaf_odd=0,
             lloyd=2, reps=4, refine=2, precision=0),
        # A whole call with host buffers and the library's default parameters
        # (8 repetitions, buckets below 200 / 400, one pass) on a set of the
        # size of the contest's dummy file.
        dict(name="contest-10k", form="host", n=10_000, d=100, k=100, data="mixture64", max_leaf=200,
             max_leaf_odd=400, lloyd=1, reps=8, refine=1, precision=0),
        # Short lists over a low-dimensional set, as small build requests ask
        # for them; an odd size.
        dict(name="short-lists-61k", form="device", n=61_003, d=64, k=10, data="subspace", max_leaf=257,
             max_leaf_odd=0, lloyd=2, reps=4, refine=2, precision=0),
        # The 100k mixture: 64 Gaussians, buckets up to 256, 8 repetitions and
        # one pass.
        dict(name="mixture-100k", form="device", n=100_000, d=100, k=100, data="mixture64", max_leaf=257,
             max_leaf_odd=0, lloyd=2, reps=8, refine=1, precision=0),
        # The same set in the precision form (BF16 estimates, FP32 re-rank).
        dict(name="mixture-100k-bf16", form="device", n=100_000, d=100, k=100, data="mixture64", max_leaf=257,
             max_leaf_odd=0, lloyd=2, reps=8, refine=1, precision=1),
        # Wide rows, lists of 50, a ragged size.
        dict(name="wide-217k", form="device", n=217_333, d=128, k=50, data="subspace", max_leaf=513, max_leaf_odd=0,
             lloyd=2, reps=3, refine=1, precision=0),
        # The headline build's schedule and distribution (subspace clusters of
        # Zipf sizes, buckets up to 1,024, 4 repetitions and 2 passes) at the
        # largest size of a served request.
        dict(name="headline-2m", form="device", n=2_000_000, d=100, k=100, data="subspace", max_leaf=1025,
             max_leaf_odd=0, lloyd=2, reps=4, refine=2, precision=0),
        # Many independent sets in one build: sizes log-uniform from 1,000 up,
        # 16-Gaussian mixtures.
        dict(name="batch-40", form="batch", sets=40, mix=2, set_lo=1000, set_hi=50_000, n=400_000, d=100, k=100,
             data="mixture16", max_leaf=1025, max_leaf_odd=0, lloyd=2, reps=4, refine=2, precision=0),
        # The KD splitter's whole build (5 repetitions, buckets below 400).
        dict(name="kd-150k", form="kd", n=150_000, d=100, k=100, data="subspace", max_leaf=400, max_leaf_odd=0,
             lloyd=0, reps=5, refine=0, precision=0),
        # The schedule driven by a recall target, host buffers.
        dict(name="adaptive-100k", form="adaptive", n=100_001, d=100, k=100, data="subspace", max_leaf=1025,
             max_leaf_odd=0, lloyd=2, reps=6, refine=4, precision=0),
        # The bucket pass on the caller's own partition (buckets of 2 to 1,024
        # points) and the finished lists: the stage calls.
        dict(name="buckets-300k", form="buckets", n=300_000, d=100, k=100, data="subspace", max_leaf=1025,
             max_leaf_odd=0, lloyd=0, reps=1, refine=0, precision=0),
        # Build requests of mixed sizes and dimensions, served side by side.
        dict(name="served-6", form="served", sets=6, mix=3, set_lo=10_000, set_hi=120_000, n=240_000, d=0, k=100,
             data="subspace", max_leaf=1025, max_leaf_odd=0, lloyd=2, reps=4, refine=2, precision=0),
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    form = rng.choice(["device", "device", "device", "device", "device", "host", "bf16", "batch", "kd", "adaptive",
                       "buckets", "served"])
    case = dict(form=form, d=rng.choice([64, 100, 100, 128]), k=rng.choice([10, 32, 50, 100, 100, 100]),
                data=rng.choice(["subspace", "mixture16", "mixture64"]), max_leaf=rng.choice([257, 513, 1025]),
                max_leaf_odd=0, lloyd=rng.choice([1, 2]), reps=rng.randint(2, 6), refine=rng.randint(0, 2),
                precision=0)
    if form == "device":
        case["n"] = _log_uniform(rng, 1000, 1_000_000)
        if case["k"] < 50 or case["n"] > 300_000:
            case["reps"] = min(case["reps"], 4)
    elif form == "bf16":
        case.update(form="device", precision=1, n=_log_uniform(rng, 10_000, 200_000))
    elif form == "host":
        case.update(n=_log_uniform(rng, 2000, 100_000), max_leaf=200, max_leaf_odd=400, lloyd=1, reps=8)
    elif form == "batch":
        sets = rng.randint(8, 60)
        case.update(sets=sets, mix=rng.randrange(1 << 16), set_lo=1000, set_hi=50_000, n=sets * 10_000)
    elif form == "kd":
        case.update(n=_log_uniform(rng, 10_000, 300_000), max_leaf=rng.choice([200, 400]), reps=5, lloyd=0,
                    refine=rng.randint(0, 1))
    elif form == "adaptive":
        case.update(n=_log_uniform(rng, 20_000, 200_000), reps=6, refine=4)
    elif form == "buckets":
        case.update(n=_log_uniform(rng, 10_000, 400_000), reps=1, refine=0, lloyd=0)
    elif form == "served":
        sets = rng.randint(3, 8)
        case.update(sets=sets, mix=rng.randrange(1 << 16), set_lo=10_000, set_hi=120_000, n=sets * 40_000, d=0, k=100)
    return case


# -------------------------------------------------------------------- inputs

def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _points(data: str, n: int, d: int, seed: int) -> torch.Tensor:
    """n x d float32 points on the device: isotropic Gaussian mixtures (sigma
    0.15 / 0.2 around centres in [-1, 1]^d) or clusters of Zipf(1.1) sizes,
    each a random 24-d subspace with noise (the headline distribution)."""
    g = _generator(seed)
    if data.startswith("mixture"):
        clusters = int(data[len("mixture"):])
        sigma = 0.15 if clusters == 64 else 0.2
        centres = torch.rand(clusters, d, generator=g, device="cuda") * 2 - 1
        labels = torch.randint(clusters, (n,), generator=g, device="cuda")
        pts = torch.randn(n, d, generator=g, device="cuda").mul_(sigma)
        return pts.add_(centres[labels])
    clusters, rank = max(8, min(1024, n // 500)), 24
    w = 1.0 / torch.arange(1, clusters + 1, device="cuda", dtype=torch.float64) ** 1.1
    sizes = torch.floor(w / w.sum() * n).to(torch.int64)
    sizes[: n - int(sizes.sum())] += 1
    a = torch.randn(clusters, d, rank, generator=g, device="cuda", dtype=torch.float64)
    chol = torch.linalg.cholesky(a.transpose(1, 2) @ a)
    basis = torch.linalg.solve_triangular(chol, a.transpose(1, 2), upper=False).float() * 0.3  # rows orthonormal
    centres = torch.rand(clusters, d, generator=g, device="cuda") * 2 - 1
    pts = torch.randn(n, d, generator=g, device="cuda").mul_(0.05)
    z = torch.randn(n, rank, generator=g, device="cuda")
    row = 0
    for c, m in enumerate(sizes.tolist()):
        block = pts[row:row + m]
        block.addmm_(z[row:row + m], basis[c])
        block.add_(centres[c])
        row += m
    return pts[torch.randperm(n, generator=g, device="cuda")]


def _sizes(case: dict) -> list[int]:
    """Sizes of a batch's sets or a stream's requests: log-uniform, adding up
    to case["n"]; a case's own, so that every seed is the same amount of work."""
    rng = np.random.default_rng(case["mix"])
    s = np.exp(rng.uniform(np.log(case["set_lo"]), np.log(case["set_hi"]), size=case["sets"]))
    s = np.maximum(case["set_lo"], np.floor(s * (case["n"] / s.sum()))).astype(np.int64)
    s[int(s.argmax())] += case["n"] - int(s.sum())
    return [int(v) for v in s]


def _buckets(case: dict, seed: int) -> np.ndarray:
    """Boundaries of consecutive buckets of 2 .. max_leaf - 1 points covering
    all n (sizes as uneven as a tree's leaves)."""
    rng = np.random.default_rng(seed)
    edges, at, n, top = [0], 0, case["n"], case["max_leaf"] - 1
    while at < n:
        b = int(min(top, max(2, rng.integers(top // 8, top + 1) if rng.random() < 0.9 else rng.integers(2, 65))))
        b = min(b, n - at)
        if n - at - b == 1:
            b = b - 1 if b > 2 else b + 1
        at += b
        edges.append(at)
    return np.asarray(edges, np.uint32)


def _params(case: dict):
    make = kd_params if case["form"] == "kd" else default_params
    return make(k=case["k"], max_leaf=case["max_leaf"], max_leaf_odd=case["max_leaf_odd"],
                lloyd_iters=max(1, case["lloyd"]), reps=case["reps"], refine=case["refine"],
                precision=case["precision"], seed=2023)


def _pinned(t: torch.Tensor) -> np.ndarray:
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()


class _Handle:
    """A context of the C ABI, for the entry points that take device buffers
    of a whole batch."""

    def __init__(self, budget: int):
        self.lib = load_library()
        self.ptr = ctypes.c_void_p()
        status = self.lib.knng_create(0, budget, ctypes.byref(self.ptr))
        if status != 0:
            raise RuntimeError("knng_create: status %d" % status)

    def check(self, status: int) -> None:
        if status != 0:
            raise RuntimeError("status %d: %s" % (status, self.lib.knng_last_error(self.ptr)))

    def __del__(self):
        if self.ptr:
            self.lib.knng_destroy(self.ptr)
            self.ptr = None


def prepare(case: dict, seed: int) -> dict:
    form, n, k = case["form"], case["n"], case["k"]
    s = dict(case=case, params=_params(case))
    if form == "served":
        rng = np.random.default_rng(case["mix"] + 1)
        s["jobs"] = [_pinned(_points(case["data"], m, int(rng.choice([64, 100, 128])), seed + 17 * i))
                     for i, m in enumerate(_sizes(case))]
        s["server"] = KnngServer(0, SERVER_BUDGET, max_running=4)
        return s
    if form == "batch":
        sizes = _sizes(case)
        s["points"] = torch.cat([_points(case["data"], m, case["d"], seed + 17 * i) for i, m in enumerate(sizes)])
        s["offsets"] = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
        s["handle"] = _Handle(CONTEXT_BUDGET)
    else:
        s["points"] = _points(case["data"], n, case["d"], seed)
        s["ctx"] = KnngContext(0, CONTEXT_BUDGET)
    if form in ("device", "batch"):
        s["ids"] = torch.empty(n, k, dtype=torch.int32, device="cuda")
        s["dists"] = torch.empty(n, k, dtype=torch.float32, device="cuda")
    else:
        s["points"] = _pinned(s["points"])
    if form == "buckets":
        edges = _buckets(case, seed)
        s["starts"], s["ends"] = edges[:-1], edges[1:]
        s["ctx"].load_points(s["points"])
    torch.cuda.synchronize()  # the points are there before a context's own stream reads them
    return s


# ----------------------------------------------------------------------- run

def run(s: dict):
    case, p = s["case"], s["params"]
    form = case["form"]
    if form == "device":
        s["ctx"].build_device(s["points"].data_ptr(), case["n"], case["d"], s["ids"].data_ptr(),
                              s["dists"].data_ptr(), p)
        return {"ids": s["ids"], "dists": s["dists"]}
    if form == "batch":
        h, st = s["handle"], Stats()
        h.check(h.lib.knng_build_batch(h.ptr, s["points"].data_ptr(), case["n"], case["d"], 4 * case["d"],
                                       s["offsets"].ctypes.data, len(s["offsets"]) - 1, 1, ctypes.byref(p),
                                       s["ids"].data_ptr(), s["dists"].data_ptr(), ctypes.byref(st)))
        return {"ids": s["ids"], "dists": s["dists"]}
    if form == "served":
        jobs = [s["server"].submit(pts, p, want_dists=True) for pts in s["jobs"]]
        out = []
        for job in jobs:
            out.extend(s["server"].result(job))
            s["server"].release(job)
        return [np.asarray(a) if a.dtype != np.uint32 else a.view(np.int32) for a in out]
    if form == "host":
        ids, dists = s["ctx"].build(s["points"], p, want_dists=True)
    elif form == "kd":
        ids, dists = s["ctx"].build_kd(s["points"], p, want_dists=True)
    elif form == "adaptive":
        ids, dists = s["ctx"].build_adaptive(s["points"], 0.95, 1000, p, want_dists=True)
    else:
        s["ctx"].reset_sets(case["k"])
        s["ctx"].begin_rep()
        s["ctx"].process_leaves(s["starts"], s["ends"])
        ids, dists = s["ctx"].finalize(want_dists=True)
    return {"ids": ids.view(np.int32), "dists": dists}


# -------------------------------------------------------------- work, exact

def work(case: dict) -> dict:
    """Bytes: the points read once, the lists written once.  Operations: per
    repetition, 3 d per unordered pair of a bucket (of 0.6 times the bound)
    and 2 d per point and tree level; per neighbour-of-neighbour pass, 2 d per
    point and candidate (k lists of k, each pair met from both ends)."""
    n, d, k = case["n"], case["d"] or 100, case["k"]
    leaf = min(n, 0.6 * case["max_leaf"])
    levels = max(0.0, math.log2(n / leaf))
    reps = min(case["reps"], 3) if case["form"] == "adaptive" else case["reps"]
    passes = min(case["refine"], 1) if case["form"] == "adaptive" else case["refine"]
    if case["form"] == "buckets":
        levels = 0.0
    flops = reps * n * (leaf / 2 * 3 * d + levels * 2 * d) + passes * n * (k * k / 2) * 2 * d
    return {"bytes": float(4 * n * d + 8 * n * k), "flops": float(flops)}


def _exact_lists(pts: torch.Tensor, k: int) -> torch.Tensor:
    """The k smallest squared distances from every point to the others, 64
    bits, ascending, padded with infinities."""
    x, m = pts.double(), pts.shape[0]
    out = torch.full((m, k), math.inf, dtype=torch.float64, device=x.device)
    for r in range(0, m, 128):
        diff = x[r:r + 128, None, :] - x[None, :, :]
        dist = diff.square_().sum(-1)
        rows = torch.arange(r, min(m, r + 128), device=x.device)
        dist[rows - r, rows] = math.inf
        kk = min(k, m)
        out[r:r + 128, :kk] = dist.topk(kk, dim=1, largest=False, sorted=True).values
    return out


def exact(case: dict, seed: int):
    if case["precision"] != 0:
        return None
    if case["form"] == "buckets":
        pts = _points(case["data"], case["n"], case["d"], seed)
        edges = _buckets(case, seed).tolist()
        dists = torch.cat([_exact_lists(pts[a:b], case["k"]) for a, b in zip(edges[:-1], edges[1:])])
        return {"ids": None, "dists": dists}
    if case["form"] in ("device", "host") and case["n"] < case["max_leaf"] and case["n"] > case["k"]:
        return {"ids": None, "dists": _exact_lists(_points(case["data"], case["n"], case["d"], seed), case["k"])}
    return None
