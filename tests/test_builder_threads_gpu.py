"""Scenes built, held and destroyed on several threads and streams at once: a build
that fails on any of them fails the test, and every comparison is counted."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import libsvo_b200 as L
from test_gpu_builder import host_pool

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [2, 4])
def test_builds_at_once(cuda, threads):
    import torch

    meshes = [(L.icosphere(3, seed=s), 7 + s % 3) for s in range(4)]
    want = [host_pool(v, t, d, 3)[1:] for (v, t), d in meshes]
    rounds = 8

    def work(k):
        stream = torch.cuda.Stream()
        alive, compared = [], 0
        for r in range(rounds):
            i = (k + r) % 4
            (v, t), d = meshes[i]
            alive.append((i, L.DeviceScene(v, t, d, treelet_levels=3, stream=stream)))
            if len(alive) > 2:
                alive.pop(0)[1].close()
            for j, ds in alive:
                n, a = ds.getIncoreBuffer()
                assert np.array_equal(n, want[j][0]) and np.array_equal(a, want[j][1]), (k, r, j)
                compared += 1
        for _, ds in alive:
            ds.close()
        return compared

    with ThreadPoolExecutor(threads) as pool:
        done = [f.result() for f in [pool.submit(work, k) for k in range(threads)]]
    assert done == [2 * rounds - 1] * threads
