"""The GPU builder where its passes split: one triangle, keys that fill and cross
blocks, columns tested again, octrees built by chunks, meshes denser than the
voxels, and several scenes alive at once -- each pool against the host path's,
record for record."""
import threading

import numpy as np
import pytest

import libsvo_b200 as L
from test_gpu_builder import assert_same, host_pool

pytestmark = pytest.mark.gpu


def shrunk(sub, radius, centre):
    v, t = L.icosphere(sub, radius=0.4, octaves=3, amplitude=0.05, frequency=2.0, seed=3)
    return (v * np.float32(radius / 0.4) + np.asarray(centre, dtype=np.float32)).astype(np.float32), t


def soup(seed, n, size):
    """Triangles of random place and shape: slivers, needles and points among
    them (no dominant axis: the whole box of the triangle is tested)."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(-0.45, 0.45, size=(n, 1, 3))
    q = p + rng.normal(size=(n, 3, 3)) * size * rng.uniform(0.01, 1.0, size=(n, 1, 1))
    k = n // 4
    s = rng.uniform(size=(k, 1))
    q[:k, 2] = q[:k, 0] * s + q[:k, 1] * (1 - s)  # on a line
    q[k:k + k // 2, 1:] = q[k:k + k // 2, :1]  # points
    q[2 * k:3 * k, :, 1] = np.round(q[2 * k:3 * k, :, 1] * 64) / 64  # on voxel planes
    return np.clip(q, -0.5, 0.5).reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("attributed", [False, True])
@pytest.mark.parametrize("n,depth,levels,size", [(1, 1, 0, 0.3), (1, 6, 2, 0.3), (3, 3, 0, 0.2), (40, 5, 2, 0.2),
                                                 (700, 6, 3, 0.1), (3000, 4, 0, 0.05), (6000, 8, 4, 0.05)])
def test_soup_matches_host(cuda, n, depth, levels, size, attributed):
    v, t = soup(n + depth, n, size)
    attrs = L.vertex_attributes(v, t, 5) if attributed else (None, None)
    try:
        L.Scene.from_mesh(v, t, depth, treelet_levels=levels, normals=attrs[0], colors=attrs[1]).close()
    except L.SvoError as refused:  # too few nodes for a treelet slot
        with pytest.raises(L.SvoError) as e:
            L.DeviceScene(v, t, depth, treelet_levels=levels, normals=attrs[0], colors=attrs[1])
        assert e.value.code == refused.code
        return
    assert_same(v, t, depth, levels, attrs)


@pytest.mark.parametrize("depth,sub,centre", [(21, 0, (0, 0, 0)), (21, 2, (0, 0, 0)), (21, 3, (0.25, -0.125, 0.0)),
                                              (20, 3, (0.25, -0.125, 0.0)), (19, 2, (0, 0, 0)), (18, 1, (-0.3, 0.2, 0.1))])
def test_chunks_match_host(cuda, depth, sub, centre):
    """Keys of more than 64 bits: the octree is built by cells of its top levels
    (all of them around the origin, one away from it); up to three of them."""
    v, t = shrunk(sub, 24.0 / 2 ** depth, centre)
    if 3 * (depth - 3) + (len(t) - 1).bit_length() > 64:
        with pytest.raises(L.SvoError) as e:
            L.DeviceScene(v, t, depth, treelet_levels=5)
        assert e.value.code == L.SVO_ERR_RANGE
        return
    assert_same(v, t, depth, 5, L.vertex_attributes(v, t, 2))
    assert_same(v, t, depth, 0)


def test_scenes_side_by_side(cuda):
    """Scenes alive, destroyed and rebuilt in turn, on two threads and streams:
    none sees another's memory."""
    import torch

    meshes = [(L.icosphere(3, seed=s), 7 + s % 2) for s in range(4)]
    want = [host_pool(v, t, d, 3)[1:] for (v, t), d in meshes]
    bad = []

    def work(k):
        stream = torch.cuda.Stream()
        alive = []
        for r in range(6):
            i = (k + r) % 4
            (v, t), d = meshes[i]
            alive.append((i, L.DeviceScene(v, t, d, treelet_levels=3, stream=stream)))
            if len(alive) > 2:
                alive.pop(0)[1].close()
            for j, ds in alive:
                n, a = ds.getIncoreBuffer()
                if not (np.array_equal(n, want[j][0]) and np.array_equal(a, want[j][1])):
                    bad.append((k, r, j))
        for _, ds in alive:
            ds.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad
