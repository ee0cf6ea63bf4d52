"""Frames, shadow frames and analysis passes at the sizes where the rays of a
warp change (up to 2^14 and 3 * 2^14 pixels) and where a grid's rows run out,
against the oracle."""
import numpy as np
import pytest

import libsvo_b200 as L
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pool(cuda, small_menger_scene):
    mm = L.TreeletMemoryManagerCuda(small_menger_scene, small_menger_scene.info.treelet_bytes)
    mm.initDeviceBuffer()
    mm.sync()
    yield mm
    mm.close()


@pytest.mark.parametrize("w,h", [(1, 1), (7, 3), (17, 2), (128, 128), (127, 129), (128, 129), (1, 16384), (16385, 1),
                                 (256, 192), (255, 193), (257, 192), (3, 70000), (1, 140001)])
def test_frames_match_the_oracle(pool, w, h):
    import torch

    nodes, attribs = pool.getIncoreBuffer()
    p = L.orbit_camera(w + h, w, h, radius=1.3).frame_params(t_scale_ratio=0.002)
    rgba = torch.zeros((h, w), dtype=torch.int32, device="cuda")
    hits = torch.zeros((h * w * 16,), dtype=torch.uint8, device="cuda")
    pool.render(p, rgba, hits)
    torch.cuda.synchronize()
    o_rgba, o_hits, _, _ = oracle.render(nodes, attribs, bytes(p))
    assert np.array_equal(rgba.cpu().numpy().view(np.uint32), o_rgba)
    assert np.array_equal(hits.cpu().numpy().view(np.uint32), np.ascontiguousarray(o_hits).view(np.uint32).reshape(-1))
    light = L.seeded_light(4)
    pool.render_shadow(p, rgba, L.shadow_cfg(light))
    torch.cuda.synchronize()
    want = oracle.render_shadow(nodes, attribs, bytes(p), light)[0]
    assert np.array_equal(rgba.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("w,h", [(1, 1), (9, 5), (128, 128), (128, 129), (255, 193), (2, 66000)])
def test_analysis_records_match_the_oracle(pool, w, h):
    import ctypes

    import torch

    nodes, _ = pool.getIncoreBuffer()
    p = L.orbit_camera(3, w, h, radius=1.4).frame_params()
    rec = torch.zeros((h * w, 4), dtype=torch.int32, device="cuda")
    d_nodes, _, n = pool.getDeviceIncoreBuffer()
    assert L.lib.svo_feedback_render(ctypes.c_void_p(d_nodes), ctypes.c_uint64(n), ctypes.byref(p), 13,
                                     ctypes.c_void_p(rec.data_ptr()), None, None) == L.SVO_OK
    torch.cuda.synchronize()
    want = oracle.feedback(nodes, bytes(p))
    want = want[0] if isinstance(want, tuple) else want
    assert np.array_equal(rec.cpu().numpy().reshape(-1).view(np.uint32), np.ascontiguousarray(want).view(np.uint32).reshape(-1))
