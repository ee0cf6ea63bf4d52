"""render_host into host memory that the program registered itself, at its edges and
across two registrations side by side, equal to the frame in pageable memory."""
import mmap

import numpy as np
import pytest

import libsvo_b200 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("w,h", [(1, 1), (64, 64), (255, 193), (640, 409)])
def test_registered_image(cuda, small_menger_scene, w, h, split):
    import torch

    mm = L.TreeletMemoryManagerCuda(small_menger_scene, small_menger_scene.info.treelet_bytes)
    mm.initDeviceBuffer()
    p = L.orbit_camera(w, w, h, radius=1.4).frame_params()
    want = mm.render_host(p)
    memory = mmap.mmap(-1, 1 << 20)
    words = np.frombuffer(memory, dtype=np.uint32)
    base, rt = words.ctypes.data, torch.cuda.cudart()
    parts = [(0, 1 << 19), (1 << 19, 1 << 19)] if split else [(0, 1 << 20)]
    for at, size in parts:
        assert int(rt.cudaHostRegister(base + at, size, 2)) == 0
    try:
        for first in sorted({0, 5, len(words) - w * h, max(0, len(words) // 2 - w * h // 2)}):
            words[:] = 7
            image = words[first:first + w * h]
            mm.render_host(p, image.reshape(h, w))
            assert np.array_equal(image.reshape(h, w), want)
            assert (words[:first] == 7).all() and (words[first + w * h:] == 7).all()
    finally:
        for at, _ in parts:
            assert int(rt.cudaHostUnregister(base + at)) == 0
        mm.close()
