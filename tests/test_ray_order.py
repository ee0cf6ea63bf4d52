"""Which kernel casts a large set of explicit rays (libsvo_b200/csrc/ray_order.cuh,
compiled for the host): sets in raster order keep a thread a ray, sets without
order have lanes take further rays."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent / "hostsim"
LIB = HERE / "_build" / "libray_order_host.so"


@pytest.fixture(scope="module")
def lib():
    src = HERE / "ray_order_host.cpp"
    deps = [src, HERE / "host_shim.h", HERE.parent.parent / "libsvo_b200" / "csrc" / "ray_order.cuh"]
    if not LIB.is_file() or any(LIB.stat().st_mtime < d.stat().st_mtime for d in deps):
        LIB.parent.mkdir(parents=True, exist_ok=True)
        subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-o", str(LIB), str(src)], check=True)
    lib = ctypes.CDLL(str(LIB))
    lib.host_close_pairs.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p]
    lib.host_close_pairs.restype = ctypes.c_uint32
    return lib


def in_order(lib, o, d):
    o, d = (np.ascontiguousarray(a, dtype=np.float32) for a in (o, d))
    last = ctypes.c_uint64()
    close = lib.host_close_pairs(o.ctypes.data, d.ctypes.data, len(o), ctypes.byref(last))
    assert last.value < len(o)
    return close >= lib.host_close_needed()


def pixel_rays(w, h, scale=1.0):
    y, x = np.mgrid[0:h, 0:w]
    d = np.stack([(x + 0.5) / w - 0.5, (y + 0.5) / h - 0.5, np.ones((h, w))], -1).reshape(-1, 3)
    return np.tile([0.3, -0.2, -1.5], (w * h, 1)), d * scale


@pytest.mark.parametrize("scale", [1e-12, 1.0, 1e12])
@pytest.mark.parametrize("w,h", [(64, 3200), (512, 512), (1023, 257), (640, 480), (4096, 64)])
def test_pixel_rays(lib, w, h, scale):
    o, d = pixel_rays(w, h, scale)
    assert in_order(lib, o, d)
    assert in_order(lib, d / scale, np.tile([0.1 * scale, 0.2 * scale, 0.3 * scale], (w * h, 1)))  # parallel rays
    mixed = np.random.default_rng(w).permutation(w * h)
    assert not in_order(lib, o[mixed], d[mixed])
    assert not in_order(lib, d[mixed] / scale, o[mixed])


@pytest.mark.parametrize("n", [16, 17, 131072, 200001])
def test_rays_without_order(lib, n):
    rng = np.random.default_rng(n)
    o, d = rng.normal(size=(2, n, 3))
    assert not in_order(lib, o, d)
    assert not in_order(lib, np.zeros((n, 3)), d)
    assert not in_order(lib, o, np.ones((n, 3)))


def test_rays_that_are_not_numbers(lib):
    o, d = pixel_rays(512, 512)
    assert not in_order(lib, o * np.nan, d)
    assert not in_order(lib, o, d * np.nan)
