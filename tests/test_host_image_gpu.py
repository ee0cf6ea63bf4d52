"""render_host into page-locked memory, which the cast writes itself: every pixel
and nothing beyond them, at sizes that cut blocks and change the rays of a warp,
in all view modes, equal to the frame in pageable memory."""
import numpy as np
import pytest

import libsvo_b200 as L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mm(cuda, small_menger_scene):
    m = L.TreeletMemoryManagerCuda(small_menger_scene, small_menger_scene.info.treelet_bytes)
    m.initDeviceBuffer()
    yield m
    m.close()


@pytest.mark.parametrize("mode", range(8))
@pytest.mark.parametrize("w,h", [(1, 1), (3, 5), (64, 64), (130, 127), (255, 193), (301, 201), (1024, 1025)])
def test_page_locked_image(mm, w, h, mode):
    import torch

    p = L.orbit_camera(w, w, h, radius=1.4).frame_params(mode=mode)
    for skip in (0, 1, 3):  # images that begin at any pixel's address
        out = torch.full((h * w + 8,), -7, dtype=torch.int32).pin_memory()
        image = out[skip:skip + h * w]
        mm.render_host(p, image)
        want = mm.render_host(p)  # pageable
        assert np.array_equal(image.numpy().view(np.uint32).reshape(h, w), want)
        assert (out[:skip] == -7).all() and (out[skip + h * w:] == -7).all()


def test_stats_and_streams(mm):
    import torch

    mm.sync()
    p = L.orbit_camera(2, 320, 200).frame_params()
    out = torch.empty((200, 320), dtype=torch.int32).pin_memory()
    s = torch.cuda.Stream()
    mm.render_host(p, out, stream=s)
    assert np.array_equal(out.numpy().view(np.uint32), mm.render_host(p))
    assert mm.sync().bounds_errors == 0
