"""Results copied to host memory: sizes around the point where several threads
carry them (2 MiB), odd last pieces, and contexts in threads side by side,
against the device-resident build's lists."""
from __future__ import annotations

import threading
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from sigmod23ann_b200 import KnngContext, default_params, workloads

pytestmark = pytest.mark.gpu

PARAMS = dict(reps=1, refine=0, max_leaf=200, max_leaf_odd=0, lloyd_iters=1, seed=4)


def _device_lists(pts: np.ndarray, k: int):
    import torch

    n, d = pts.shape
    x = torch.from_numpy(pts).cuda()
    ids = torch.empty(n, k, dtype=torch.int32, device="cuda")
    dist = torch.empty(n, k, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    with KnngContext(0) as c:
        c.build_device(x.data_ptr(), n, d, ids.data_ptr(), dist.data_ptr(), default_params(k=k, **PARAMS))
    return ids.cpu().numpy().view(np.uint32), dist.cpu().numpy()


# 2 MiB of 4-byte entries: n k = 524,288.
@pytest.mark.parametrize("n,k", [(5242, 100), (5243, 100), (20_973, 100), (65_536, 32), (50_001, 77), (90_000, 100)])
def test_lists_equal_the_device_resident_ones(knng_lib, n, k):
    pts = workloads.gaussian_mixture(n=n, d=64, clusters=16, sigma=0.2, seed=n)
    want_ids, want_dist = _device_lists(pts, k)
    with KnngContext(0) as c:
        for _ in range(2):
            ids, dist = c.build(pts, default_params(k=k, **PARAMS), want_dists=True)
            assert np.array_equal(ids, want_ids)
            assert np.array_equal(dist.view(np.uint32), want_dist.view(np.uint32))


def test_contexts_in_threads(knng_lib):
    sets = [workloads.gaussian_mixture(n=22_000 + 1000 * i, d=64, clusters=8, sigma=0.2, seed=i) for i in range(4)]
    want = [_device_lists(p, 100)[0] for p in sets]
    bad = []

    def work(i: int) -> None:
        for _ in range(2):
            with KnngContext(0, 4 << 30) as c:
                if not np.array_equal(c.build(sets[i], default_params(k=100, **PARAMS)), want[i]):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_every_thread_finishes_its_builds(knng_lib):
    """Contexts in threads as above, with distances, each build's outcome looked at:
    an error in a thread fails the test."""
    sets = [workloads.gaussian_mixture(n=22_000 + 1000 * i, d=64, clusters=8, sigma=0.2, seed=i) for i in range(4)]
    want = [_device_lists(p, 100) for p in sets]

    def work(i: int) -> int:
        done = 0
        for _ in range(3):
            with KnngContext(0, 4 << 30) as c:
                for _ in range(2):
                    ids, dist = c.build(sets[i], default_params(k=100, **PARAMS), want_dists=True)
                    assert np.array_equal(ids, want[i][0]), i
                    assert np.array_equal(dist.view(np.uint32), want[i][1].view(np.uint32)), i
                    done += 1
        return done

    with ThreadPoolExecutor(4) as pool:
        assert [f.result() for f in [pool.submit(work, i) for i in range(4)]] == [6] * 4
