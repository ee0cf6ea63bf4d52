"""The traversal as the GPU runs it (packed FP32 pairs, sums rounded down, a product
by a one from constant memory that keeps a sum of products in two roundings) in
octrees as deep as it takes, against the oracle.  The same rays run through its host
stand-ins in test_traverse_paths.py."""
import numpy as np
import pytest

import libsvo_b200 as L
import oracle
from rays import edge_rays
from test_stream_rays_gpu import LINE, launch, same
from test_traverse_paths import rays_at, sparse_pool

pytestmark = pytest.mark.gpu


def check_all(nodes, o, d, tsr, S, flat):
    """Few rays (the packed loop) and many (the loop that takes further rays)."""
    import torch

    o, d = np.ascontiguousarray(o, dtype=np.float32), np.ascontiguousarray(d, dtype=np.float32)
    want, _ = oracle.cast_rays(nodes, o, d, tsr, flat=flat, stack_size=S)
    times = -(-LINE // len(o))
    for k in (1, times):
        hits, keep = launch(torch, nodes, np.tile(o, (k, 1)), np.tile(d, (k, 1)), tsr, L.trace_cfg(int(flat), S))
        torch.cuda.synchronize()
        assert same(hits, np.tile(want, k)), f"stack size {S}, {k * len(o)} rays"
    return want


@pytest.mark.parametrize("depth", [13, 16, 18, 20, 21, 22, 23])
def test_treelet_rules(cuda, depth):
    rng = np.random.default_rng(depth)
    nodes, c = sparse_pool(depth, depth, 400)
    o, d = rays_at(rng, np.concatenate([c] * 8))
    eo, ed = edge_rays(n_random=1500, seed=depth)
    o, d = np.concatenate([o, eo]), np.concatenate([d, ed])
    for S in sorted({depth - 1, depth, depth + 1, 24}):
        h = check_all(nodes, o, d, 0.0, S, False)
        # voxels smaller than the rules' epsilon of 1e-5 are walked, and rarely hit
        assert h["loops"].mean() > depth
    for tsr in (1e-6, 0.001):
        check_all(nodes, o, d, tsr, 24, False)


@pytest.mark.parametrize("depth", [13, 16, 20, 22, 23, 24])
def test_flat_rules(cuda, depth):
    rng = np.random.default_rng(depth)
    nodes, c = sparse_pool(depth, depth, 400, absolute=True)
    o, d = rays_at(rng, np.concatenate([c] * 8))
    for S in sorted({depth - 1, depth, 24}):
        h = check_all(nodes, o, d, 0.0, S, True)
        assert h["loops"].mean() > depth
