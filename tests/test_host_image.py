"""Which host images the cast writes itself (libsvo_b200/csrc/host_image.cpp), over
registrations that the host pretends (tests/hostsim/host_image_host.cpp): only those
that registrations hold from the first byte to the last."""
import ctypes
import os
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent / "hostsim"
SOURCE = HERE.parent.parent / "libsvo_b200" / "csrc" / "host_image.cpp"
CUDA_HOME = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
HOST, DEVICE, MANAGED = 1, 2, 3
PAGE = 4096


def load(source, tag):
    lib = HERE / "_build" / f"libhost_image_{tag}.so"
    lib.parent.mkdir(parents=True, exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", f"-I{CUDA_HOME / 'include'}",
                    f'-DHOST_IMAGE_SOURCE="{source}"', "-o", str(lib), str(HERE / "host_image_host.cpp")], check=True)
    lib = ctypes.CDLL(str(lib))
    u64 = ctypes.c_uint64
    lib.registered.argtypes = [u64, u64, ctypes.c_int]
    lib.mapped.argtypes, lib.mapped.restype = [u64, u64], u64
    return lib


@pytest.fixture(scope="module")
def lib():
    lib = load(SOURCE, "here")
    lib.registered(16 * PAGE, 4 * PAGE, HOST)
    lib.registered(32 * PAGE, PAGE, HOST)  # two with pageable memory between them
    lib.registered(34 * PAGE, PAGE, HOST)
    lib.registered(64 * PAGE, PAGE, HOST)  # two side by side
    lib.registered(65 * PAGE, PAGE, HOST)
    lib.registered(96 * PAGE, PAGE, DEVICE)
    lib.registered(128 * PAGE, PAGE, MANAGED)
    return lib


@pytest.mark.parametrize("at,pixels", [(16 * PAGE, 1), (16 * PAGE, PAGE), (16 * PAGE + 4, PAGE - 1),
                                       (17 * PAGE, PAGE // 4), (20 * PAGE - 4, 1), (32 * PAGE, PAGE // 4),
                                       (64 * PAGE, PAGE // 2), (65 * PAGE - 4, 2), (64 * PAGE + 8, PAGE // 2 - 2)])
def test_images_that_the_cast_writes(lib, at, pixels):
    assert lib.mapped(at, pixels) == at


@pytest.mark.parametrize("at,pixels", [
    (32 * PAGE, 3 * PAGE // 4),  # first and last pixel registered, pageable memory between
    (33 * PAGE - 4, PAGE // 4 + 2),
    (64 * PAGE, PAGE // 2 + 1),
    (16 * PAGE, PAGE + 1), (16 * PAGE + 4, PAGE), (20 * PAGE - 4, 2),  # its end lies beyond
    (15 * PAGE, PAGE // 2), (8 * PAGE, 4),  # its beginning, or all of it
    (16 * PAGE + 2, 1), (16 * PAGE + 1, 8),  # between pixels
    (96 * PAGE, 4), (128 * PAGE, 4),  # not host memory
    (16 * PAGE, 1 << 62), (16 * PAGE, (1 << 64) - 1)])
def test_images_that_are_copied_to(lib, at, pixels):
    assert lib.mapped(at, pixels) == 0


def test_without_the_drivers_answer():
    lib = load(SOURCE, "no_driver")
    lib.registered(16 * PAGE, 4 * PAGE, HOST)
    lib.no_driver()
    assert lib.mapped(16 * PAGE, 1) == 0
