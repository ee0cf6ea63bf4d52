"""The traversal's two loops (the general one of every ray, the fast one of rays
with finite reciprocals) and the step from one to the other, as compiled for the
host, against the oracle: every stack size, pools with nodes outside, rays
through cell edges and corners, and rays that never end."""
import numpy as np
import pytest

import libsvo_b200 as L
import oracle
from rays import edge_rays, random_octree_pool
from test_traverse_host import check, host_lib  # noqa: F401


def sparse_pool(seed, depth, leaves, absolute=False):
    """A breadth-first pool of an octree with about `leaves` leaves at `depth`
    (any depth up to 24), and the leaves' centres."""
    rng = np.random.default_rng(seed)
    paths = rng.integers(0, 8, size=(leaves, depth))
    paths[: leaves // 2, : depth - 2] = paths[0, : depth - 2]  # half of them in one corner
    levels = []
    keys = [tuple(p) for p in paths]
    for k in range(depth + 1):
        levels.append(sorted({p[:k] for p in keys}))
    index, n = {}, 0
    for lv in levels:
        for p in lv:
            index[p] = n
            n += 1
    nodes = np.zeros((n, 2), dtype=np.uint32)
    for k, lv in enumerate(levels[:-1]):
        for p in lv:
            kids = [c for c in range(8) if p + (c,) in index]
            i = index[p]
            nodes[i, 0] = index[p + (kids[0],)] - (0 if absolute else i)
            m = sum(1 << c for c in kids)
            nodes[i, 1] = (m << 8) | (m if k + 1 == depth else 0)
    centres = np.full((leaves, 3), -0.5)
    for k in range(depth):
        for a in range(3):
            centres[:, a] += ((paths[:, k] >> (2 - a)) & 1) * 0.5 ** (k + 1)
    return nodes, centres + 0.5 ** (depth + 1)


def rays_at(rng, targets):
    o = rng.normal(size=targets.shape)
    o *= rng.uniform(0.1, 2.0, size=(len(o), 1)) / np.linalg.norm(o, axis=1, keepdims=True)
    d = targets - o
    return o, d / np.linalg.norm(d, axis=1, keepdims=True)


@pytest.mark.parametrize("depth", [2, 3, 5, 8, 13, 16, 20, 22, 23])
def test_every_depth(host_lib, depth):  # noqa: F811
    rng = np.random.default_rng(depth)
    nodes, c = sparse_pool(depth, depth, 200)
    o, d = rays_at(rng, np.concatenate([c] * 5))
    eo, ed = edge_rays(n_random=500, seed=depth)
    o, d = np.concatenate([o, eo]), np.concatenate([d, ed])
    for S in sorted({2, max(2, depth - 1), depth, depth + 1, 24}):  # at, above and below the octree's depth
        for tsr in (0.0, 0.001):
            check(host_lib, nodes, o, d, tsr, stack_size=S)


@pytest.mark.parametrize("depth", [2, 3, 8, 16, 22, 23, 24])
def test_every_depth_flat(host_lib, depth):  # noqa: F811
    rng = np.random.default_rng(depth)
    nodes, c = sparse_pool(depth, depth, 200, absolute=True)
    o, d = rays_at(rng, np.concatenate([c] * 5))
    for S in sorted({2, max(2, depth - 1), depth, 24}):  # a smaller depth ends at an inner node
        check(host_lib, nodes, o, d, 0.0, stack_size=S, flat=True)


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("seed", range(3))
def test_nodes_outside_the_pool(host_lib, seed, flat):  # noqa: F811
    rng = np.random.default_rng(seed)
    nodes, _ = random_octree_pool(seed, depth=5)
    nodes = nodes.copy()
    if flat:
        nodes[:, 0] += np.arange(len(nodes), dtype=np.uint32)
    inner = np.nonzero(nodes[:, 1] & ~(nodes[:, 1] << 8) & 0xFF00)[0][1:]
    bad = rng.choice(inner, size=len(inner) // 10 + 1, replace=False)
    nodes[bad, 0] = rng.integers(len(nodes), 2**32, size=len(bad), dtype=np.uint64).astype(np.uint32)
    o, d = edge_rays(n_random=4000, seed=seed)
    h = check(host_lib, nodes, o, d, 0.0, stack_size=5 if flat else 13, flat=flat)
    assert (h["flags"] == L.HITFLAG_BOUNDS).any()


def test_rays_through_edges_and_corners(host_lib):  # noqa: F811
    """Exits of a child and its parent through the same plane, through two or
    three planes at once, and within the reference's epsilon of each other."""
    rng = np.random.default_rng(3)
    n = 6000
    targets = rng.integers(-32, 33, size=(n, 3)) / 64.0
    dirs = rng.integers(-3, 4, size=(n, 3)).astype(np.float64)
    dirs[(dirs == 0).all(axis=1)] = 1.0
    dirs[::3] += rng.normal(size=dirs[::3].shape) * 1e-5
    o = targets - 2.0 * dirs
    d = dirs / np.linalg.norm(dirs, axis=1, keepdims=True)
    for seed in range(3):
        nodes, _ = random_octree_pool(seed, depth=6, fill=0.3)
        check(host_lib, nodes, o, d, 0.0)
        nodes[:, 0] += np.arange(len(nodes), dtype=np.uint32)
        check(host_lib, nodes, o, d, 0.0, stack_size=6, flat=True)


@pytest.mark.parametrize("scale", [1e3, 1e6, 1e30, 1e38, np.inf, np.nan])
def test_unusual_origins(host_lib, scale):  # noqa: F811
    rng = np.random.default_rng(1)
    nodes, _ = random_octree_pool(1, depth=5)
    o = rng.normal(size=(400, 3)) * scale
    o[::2, 0] = 0.1
    o[::5, 1:] = rng.normal(size=(80, 2)) * 0.2
    d = rng.normal(size=(400, 3))
    d[::3] = -np.nan_to_num(o[::3], nan=1.0, posinf=1.0, neginf=-1.0)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[::7] *= 1e-30
    check(host_lib, nodes, o, d, 0.0)


def test_rays_that_never_end(host_lib):  # noqa: F811
    """Rays the watchdog stops: the cycle they repeat is skipped from wherever
    the fast loop saw them stop advancing."""
    nodes, c = sparse_pool(9, 20, 400)
    rng = np.random.default_rng(9)
    # voxels far smaller than the reference's epsilon, from afar
    o, d = rays_at(rng, np.concatenate([c + rng.normal(size=c.shape) * 1e-6 for _ in range(20)]))
    got = check(host_lib, nodes, o * 3.0, d, 0.0, stack_size=24)
    assert oracle.FLAG_CAPPED == L.HITFLAG_CAPPED
    from libsvo_b200 import scenes
    wl = scenes.icosphere(subdivisions=5, depth=10, treelet_levels=5, width=800, height=450)
    info = wl.scene.info
    mm = L.TreeletMemoryManagerCuda(wl.scene, info.treelet_bytes * info.num_treelets)
    mm.insertAll()
    nodes, _ = mm.getIncoreBuffer()
    capped = 0
    for k in range(4):
        p = scenes.orbit_pose(2.5 - 0.3 * k, 40.0 * k + 11.0, 10.0 * k - 20.0, 800, 450, 30.0).frame_params()
        o, d = oracle.pixel_rays(bytes(p))
        h = check(host_lib, nodes, o, d, p.t_scale_ratio)
        capped += int((h["flags"] == L.HITFLAG_CAPPED).sum())
    assert capped + int((got["flags"] == L.HITFLAG_CAPPED).sum()) > 0
