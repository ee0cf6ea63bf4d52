"""The GPU builder's plan of cells (libsvo_b200/csrc/chunk_plan.h) on the host, over
boxes of columns: no cell has more than it may while it can be split, none is built
without memory for it, and together they are the octree in Morton order.  And the tests' own shortcut to a
sliver's voxels, against the host builder."""
import ctypes

import numpy as np
import pytest

import builder_host
import libsvo_b200 as L


@pytest.fixture(scope="module")
def lib():
    return builder_host.load()


def plan(lib, boxes, depth, level, max_columns, memory=1 << 62):
    b = np.ascontiguousarray(boxes, dtype=np.int32)
    out = np.zeros((512, 4), dtype=np.uint64)
    n = lib.plan(b.ctypes.data_as(ctypes.c_void_p), len(b), depth, level, max_columns, memory,
                 out.ctypes.data_as(ctypes.c_void_p), len(out))
    return out[:n].astype(np.int64) if n >= 0 else int(n)


def boxes_in(rng, n, lo, hi, longest):
    a = rng.integers(lo, hi, size=(n, 3))
    b = np.minimum(a + rng.integers(0, longest, size=(n, 3)), hi - 1)
    return np.concatenate([a, b], axis=1)


CASES = {
    "spread": (6, 0, lambda rng: boxes_in(rng, 40, 0, 64, 20)),
    "one octant": (6, 0, lambda rng: boxes_in(rng, 40, 33, 63, 20)),
    "one octant, keys of more than 64 bits": (7, 2, lambda rng: boxes_in(rng, 40, 65, 127, 40)),
    "slivers": (9, 0, lambda rng: np.array([[0, 0, 0, 511, 511, 511], [256, 256, 256, 400, 500, 510]])),
    "a pile in one voxel": (5, 1, lambda rng: np.tile([7, 9, 11, 7, 9, 11], (300, 1))),
    "one level": (1, 0, lambda rng: np.tile([0, 0, 0, 1, 1, 1], (300, 1))),
}


def built_cells(lib, name, max_columns, memory):
    depth, level, make = CASES[name]
    boxes = make(np.random.default_rng(5))
    cells = plan(lib, boxes, depth, level, max_columns, memory)
    return depth, boxes, cells


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("max_columns", [1, 60, 700, 1 << 40])
def test_cells_with_many_columns_are_split(lib, name, max_columns):
    depth, boxes, cells = built_cells(lib, name, max_columns, 1 << 62)
    last = (cells[:, 0] == 3) | (cells[:, 0] + 1 == depth)
    assert (cells[~last, 2] <= max_columns).all() and (cells[:, 0] <= 3).all()
    # cells in Morton order, each behind the one before
    begin = cells[:, 1] << (3 * (depth - cells[:, 0]))
    end = begin + (1 << (3 * (depth - cells[:, 0])))
    assert (begin[1:] >= end[:-1]).all()
    # a voxel of every box is in one of them
    for lo in boxes[:, :3]:
        code = sum(((int(lo[k]) >> b) & 1) << (3 * b + 2 - k) for b in range(depth) for k in range(3))
        assert ((begin <= code) & (code < end)).sum() == 1
    # the level at which two cells' codes part
    for i in range(1, len(cells)):
        digits = [[(int(c) >> (3 * (depth - d))) & 7 for d in range(1, depth + 1)] for c in begin[[i - 1, i]]]
        assert cells[i, 3] == 1 + next(d for d in range(depth) if digits[0][d] != digits[1][d])


@pytest.mark.parametrize("memory", [50, 400, 3000])
def test_cells_without_memory_are_split(lib, memory):
    depth, boxes, cells = built_cells(lib, "spread", 1 << 40, memory)
    whole = plan(lib, boxes, depth, 0, 1 << 40)
    assert len(whole) == 1 and whole[0, 2] > memory
    third = plan(lib, boxes, depth, 3, 1 << 40)
    if isinstance(cells, int):  # too little even for a cell of the third level
        assert cells == L.SVO_ERR_NOMEM and third[:, 2].max() > memory
    else:
        assert (cells[:, 2] <= memory).all() and cells[:, 0].max() <= 3


@pytest.mark.parametrize("depth", [8, 10, 11])
def test_near_voxels_are_the_host_builders(lib, depth):
    rng = np.random.default_rng(depth)
    for corner in ((-0.4, -0.45, -0.3), (0.01, 0.02, 0.03)):
        t = builder_host.sliver(corner, 0.4, depth, rng)
        nodes, _ = L.Scene.from_mesh(t, [[0, 1, 2]], depth, treelet_levels=0).flatten()
        nodes = nodes.copy()
        nodes[:, 0] -= np.where(nodes[:, 0] != 0, np.arange(len(nodes)), 0).astype(np.uint32)  # relative
        want = builder_host.leaves(nodes, depth)[0]
        assert np.array_equal(builder_host.near_voxels(lib, t, depth), want)
        assert len(want) > 2 ** depth * 0.4
