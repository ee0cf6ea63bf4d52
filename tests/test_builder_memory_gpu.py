"""GPU builds where device memory is short: what is held per column of voxels is
bounded, and a build whose keys do not fit at once goes on by smaller cells."""
import numpy as np
import pytest

import builder_host
import libsvo_b200 as L

pytestmark = pytest.mark.gpu
GB = 1 << 30


class only:
    """Leaves `free` bytes of the device's memory; the rest is held, not touched."""

    def __init__(self, free):
        self.free = free

    def __enter__(self):
        import torch

        torch.cuda.empty_cache()
        self.held = torch.empty(torch.cuda.mem_get_info()[0] - self.free, dtype=torch.uint8, device="cuda")

    def __exit__(self, *a):
        import torch

        del self.held
        torch.cuda.empty_cache()


def test_slivers_need_no_memory_for_their_boxes(cuda):
    """Twenty thousand triangles about a voxel wide and a thousand long in one cell of
    the third level: 10^10 columns in their boxes, which at 4 bytes each are more
    than there is, and some ten thousand voxels.  (Longer ones are beyond what FP32
    tells apart: the plane of a triangle N voxels long and one wide is off by
    N^2 / 2^24 voxels at its end.)"""
    depth = 13
    rng = np.random.default_rng(4)
    lib = builder_host.load()
    meshes, want = [], np.zeros(0, dtype=np.uint64)
    for _ in range(40):
        t = builder_host.sliver(rng.uniform(0.001, 0.002, 3), 0.12, depth, rng)
        meshes.append(t)
        want = np.union1d(want, builder_host.near_voxels(lib, t, depth))
    assert len(want) > 10000
    v = np.concatenate(meshes)
    t = np.tile(np.arange(len(v), dtype=np.uint32).reshape(-1, 3), (500, 1))
    with only(12 * GB):
        ds = L.DeviceScene(v, t, depth, treelet_levels=0)
        got, _ = ds.getIncoreBuffer()
        ds.close()
    assert np.array_equal(builder_host.leaves(got, depth)[0], want)


def test_columns_taken_in_passes_keep_their_triangles_in_order(cuda):
    """A sphere's triangles 256 times over, 6e8 columns: inside one cell of the third
    level they are walked in two passes, around a corner of eight cells in one pass a
    cell.  The vertices are on a grid on which both places are exact, so the leaves
    and their attributes, sums over the triangles in order, are the same."""
    depth = 13
    v, t = L.icosphere(2, radius=0.4, octaves=3, amplitude=0.05, frequency=2.0, seed=5)
    v = np.round(v / 8 * 2 ** 16) / 2 ** 16
    t = np.tile(t, (256, 1))

    def leaves(centre):
        ds = L.DeviceScene((v + centre).astype(np.float32), t, depth, treelet_levels=0)
        nodes, attribs = ds.getIncoreBuffer()
        pairs = ds.counts()[1]
        ds.close()
        codes, at = builder_host.leaves(nodes, depth)
        xyz = np.zeros((len(codes), 3), dtype=np.int64)
        for b in range(depth):
            for k in range(3):
                xyz[:, k] |= ((codes >> np.uint64(3 * b + 2 - k)) & np.uint64(1)).astype(np.int64) << b
        xyz -= int(centre * 2 ** depth)
        order = np.lexsort(xyz.T)
        return xyz[order], attribs[at][order], pairs

    one, eight = leaves(0.0625), leaves(0.125)
    assert one[2] == eight[2] and one[2] > 3e8
    assert np.array_equal(one[0], eight[0]) and np.array_equal(one[1], eight[1])


@pytest.mark.parametrize("attributed", [False, True])
def test_keys_that_do_not_fit_at_once(cuda, attributed):
    """Every triangle fifty times: 3.2 GB of keys and their copy for a pool of
    150 MB.  With 2 GB of memory the octree is built by its octants."""
    v, t = L.icosphere(4, radius=0.4, octaves=3, amplitude=0.05, frequency=2.0, seed=2)
    t = np.repeat(t, 50, axis=0)
    attrs = dict(zip(("normals", "colors"), L.vertex_attributes(v, t, 3))) if attributed else {}

    def pool():
        ds = L.DeviceScene(v, t, 10, treelet_levels=5, **attrs)
        out = (*ds.getIncoreBuffer(), ds.counts(), ds.info.leaf_voxels)
        ds.close()
        return out

    want = pool()
    assert want[2][1] > 150_000_000
    with only(2 * GB):
        got = pool()
    assert got[2:] == want[2:]
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
