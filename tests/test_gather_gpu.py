"""The page-locked gather: what crosses PCIe is the records a slot holds and the
single records that leaf writes changed, and the device pool still equals the
mirror -- slots taken over by smaller treelets, uploads of leaf writes alone,
more leaf writes than are listed, and slot sizes of an odd number of records."""
import numpy as np
import pytest

import libsvo_b200 as L
from test_upload_gpu import children, device_pool

pytestmark = pytest.mark.gpu


def assert_mirrored(mm):
    mm.updateDeviceMemory()
    hn, ha = mm.getIncoreBuffer()
    dn, da = device_pool(mm)
    assert np.array_equal(dn, hn) and np.array_equal(da, ha)


@pytest.mark.parametrize("extra", [0, 8, 16, 24])
def test_pool_follows_mirror(cuda, extra):
    v, t = L.icosphere(3, seed=2)
    nat = L.Scene.from_mesh(v, t, 7, treelet_levels=3).info.treelet_bytes
    scene = L.Scene.from_mesh(v, t, 7, treelet_levels=3, treelet_bytes=nat + extra)
    n = scene.info.num_treelets
    kids = children(scene)
    mm = L.TreeletMemoryManagerCuda(scene, scene.info.treelet_bytes * (n // 2))
    mm.setUploadPolicy(L.UPLOAD_PINNED)
    mm.insertAll()
    mm.initDeviceBuffer()
    assert_mirrored(mm)
    resident = [g for g in range(1, n) if mm.getSlotGid(g) >= 0]
    childless = [g for g in resident if not any(mm.getSlotGid(c) >= 0 for c in kids.get(g, []))]
    rng = np.random.default_rng(extra)
    # leaf writes alone
    for g in childless[::3]:
        assert mm.removeTreeletFromIncoreBuffer(g)
    assert mm.updateDeviceMemory() == 1
    assert_mirrored(mm)
    assert mm.updateDeviceMemory() == 0  # nothing left to bring over
    # their slots taken over by treelets of other sizes
    out = [g for g in range(1, n) if mm.getSlotGid(g) < 0 and mm.getSlotGid(scene.treelet(g)["parent_gid"]) >= 0]
    for g in rng.permutation(out).tolist():
        if mm.info.free_slots == 0:
            break
        assert mm.insertTreeletIntoIncoreBuffer(g)
    assert_mirrored(mm)
    # the same leaves over and over, uploaded once
    one = next(g for g in range(1, n) if mm.getSlotGid(g) >= 0 and
               not any(mm.getSlotGid(c) >= 0 for c in kids.get(g, [])))
    for _ in range(2500):
        assert mm.removeTreeletFromIncoreBuffer(one) and mm.insertTreeletIntoIncoreBuffer(one)
    assert mm.removeTreeletFromIncoreBuffer(one)
    assert_mirrored(mm)
    # a reset brings every slot over again, then single changes on top of it
    mm.resetIncoreBuffer()
    assert_mirrored(mm)
    first = [g for g in range(1, n) if scene.treelet(g)["parent_gid"] == 0][:5]
    for g in first:
        assert mm.insertTreeletIntoIncoreBuffer(g)
        assert_mirrored(mm)
    # another policy after the gather's lists were used
    mm.setUploadPolicy(L.UPLOAD_COALESCED)
    for g in first[1:]:
        assert mm.removeTreeletFromIncoreBuffer(g)
    assert_mirrored(mm)
    mm.close()
