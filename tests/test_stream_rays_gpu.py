"""Explicit rays in numbers where lanes take further rays (2^17 and more): rays of
every kind and length beside one another, every count around the line, two
streams at once and a captured launch, against the oracle."""
import numpy as np
import pytest

import libsvo_b200 as L
import oracle
from rays import edge_rays, random_octree_pool

pytestmark = pytest.mark.gpu
LINE = 1 << 17


def make(seed, n, depth=6):
    nodes, _ = random_octree_pool(seed, depth=depth, fill=0.3)
    o, d = edge_rays(n_random=n, seed=seed)
    rng = np.random.default_rng(seed)
    k = len(o)
    o[k // 2::11] = rng.normal(size=o[k // 2::11].shape) * 3.0  # many of these miss the root box
    d[5::97, 1] = 0.0  # the general loop
    o[7::101, 0] = -0.0
    d[3::89] *= 1e-30
    perm = rng.permutation(k)[:n]
    return nodes, np.ascontiguousarray(o[perm]), np.ascontiguousarray(d[perm])


def launch(torch, nodes, o, d, tsr, cfg, stats=None, stream=None):
    dn = torch.from_numpy(nodes.view(np.int32)).cuda()
    do, dd = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    hits = torch.full((len(o), 4), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    L.trace_rays(dn, len(nodes), do, dd, len(o), tsr, hits, cfg=cfg, d_stats=stats, stream=stream)
    return hits, (dn, do, dd)


def same(hits, want):
    return np.array_equal(hits.cpu().numpy().reshape(-1).view(np.uint32), np.ascontiguousarray(want).view(np.uint32).reshape(-1))


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("n", [LINE - 1, LINE, LINE + 1, LINE + 31, 2 * LINE + 77, 700001])
def test_rays_match_the_oracle(cuda, n, flat):
    import torch

    nodes, o, d = make(n % 7, n)
    if flat:
        nodes = nodes + np.stack([np.arange(len(nodes)), np.zeros(len(nodes))], axis=1).astype(np.uint32)
    S = 6 if flat else 13
    want, _ = oracle.cast_rays(nodes, o, d, 0.001, flat=flat, stack_size=S)
    stats = torch.zeros(4, dtype=torch.int32, device="cuda")
    hits, _ = launch(torch, nodes, o, d, 0.001, L.trace_cfg(int(flat), S), stats)
    torch.cuda.synchronize()
    assert same(hits, want)
    assert int(stats[0]) == int((want["flags"] == L.HITFLAG_CAPPED).sum())


@pytest.mark.parametrize("n", [1, 7, 9, 31, 33, (1 << 14) - 1, 1 << 14, (1 << 14) + 1, 1 << 15, (1 << 15) + 1])
def test_few_rays_match_the_oracle(cuda, n):
    """Counts cast with 8, 16 and 32 rays a warp."""
    import torch

    nodes, o, d = make(n % 5, n)
    want, _ = oracle.cast_rays(nodes, o, d, 0.001)
    hits, _ = launch(torch, nodes, o, d, 0.001, L.trace_cfg())
    torch.cuda.synchronize()
    assert same(hits, want)


def test_every_ray_misses(cuda):
    import torch

    nodes, o, d = make(1, LINE + 5)
    o[:] = 5.0
    d[:] = np.array([1.0, 0.0, 0.0], dtype=np.float32)
    want, _ = oracle.cast_rays(nodes, o, d, 0.0)
    hits, _ = launch(torch, nodes, o, d, 0.0, L.trace_cfg())
    torch.cuda.synchronize()
    assert same(hits, want)


def test_two_streams_at_once(cuda):
    import torch

    sets = [make(s, LINE + 1000 * s) for s in (2, 3)]
    want = [oracle.cast_rays(n, o, d, 0.0)[0] for n, o, d in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    for _ in range(4):
        out = [launch(torch, n, o, d, 0.0, L.trace_cfg(), stream=s) for (n, o, d), s in zip(sets, streams)]
        torch.cuda.synchronize()
        for (hits, _), w in zip(out, want):
            assert same(hits, w)


def test_captured_launch(cuda):
    import torch

    nodes, o, d = make(4, LINE + 9)
    want, _ = oracle.cast_rays(nodes, o, d, 0.0)
    hits, (dn, do, dd) = launch(torch, nodes, o, d, 0.0, L.trace_cfg())
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        L.trace_rays(dn, len(nodes), do, dd, len(o), 0.0, hits, stream=torch.cuda.current_stream())
    hits.fill_(-1)
    g.replay()
    torch.cuda.synchronize()
    assert same(hits, want)
