"""Large sets of explicit rays, in order and not: each ray is cast once, by the one
kernel or the other, and has the oracle's record."""
import numpy as np
import pytest

import libsvo_b200 as L
import oracle
from rays import random_octree_pool

pytestmark = pytest.mark.gpu
LINE = 3 << 16  # from here on the rays are asked for their order


def cast(nodes, o, d, flat=False, stream=None):
    import torch

    n = len(o)
    dn = torch.from_numpy(nodes.view(np.int32)).cuda()
    do, dd = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    hits = torch.full((n + 1, 4), -1, dtype=torch.int32, device="cuda")
    stats = torch.zeros(4, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    L.trace_rays(dn, len(nodes), do, dd, n, 0.001, hits, cfg=L.trace_cfg(int(flat), 6 if flat else 13), d_stats=stats,
                 stream=stream)
    torch.cuda.synchronize()
    got = hits.cpu().numpy()
    assert (got[n] == -1).all()
    return got[:n], stats.cpu().numpy()


def pixel_rays(n, w=1021):
    i = np.arange(n)
    d = np.stack([(i % w) / w - 0.5, (i // w) / (n // w + 1) - 0.5, np.full(n, 1.2)], -1)
    return np.tile(np.float32([0.13, -0.07, -1.4]), (n, 1)), d.astype(np.float32)


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("order", ["pixels", "mixed", "half"])
@pytest.mark.parametrize("n", [LINE - 1, LINE, LINE + 1, LINE + 127, 655361])
def test_each_ray_is_cast_once(cuda, n, order, flat):
    nodes, _ = random_octree_pool(n % 5, depth=6, fill=0.3)
    if flat:
        nodes = nodes + np.stack([np.arange(len(nodes)), np.zeros(len(nodes))], axis=1).astype(np.uint32)
    o, d = pixel_rays(n)
    p = np.arange(n)
    if order != "pixels":
        k = n if order == "mixed" else n // 2
        p[:k] = np.random.default_rng(n).permutation(k)
    o, d = np.ascontiguousarray(o[p]), np.ascontiguousarray(d[p])
    want, _ = oracle.cast_rays(nodes, o, d, 0.001, flat=flat, stack_size=6 if flat else 13)
    got, stats = cast(nodes, o, d, flat)
    assert np.array_equal(got.reshape(-1).view(np.uint32), np.ascontiguousarray(want).view(np.uint32).reshape(-1))
    assert int(stats[0]) == int((want["flags"] == L.HITFLAG_CAPPED).sum())
