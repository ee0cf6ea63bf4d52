"""The device memory that builds keep (libsvo_b200/csrc/kept_memory.cpp), over a
device that the host pretends to be (tests/hostsim/kept_memory_host.cpp): who gets
it back, when, and who waits for whom."""
import ctypes
import os
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent / "hostsim"
SOURCE = HERE.parent.parent / "libsvo_b200" / "csrc" / "kept_memory.cpp"
CUDA_HOME = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
GB = 1 << 30


def load(path, tag):
    """The pretended device with the given source, in a library of its own."""
    lib = HERE / "_build" / f"libkept_memory_{tag}.so"
    lib.parent.mkdir(parents=True, exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-pthread", "-Wl,-Bsymbolic", f"-I{CUDA_HOME / 'include'}",
                    f'-DKEPT_MEMORY_SOURCE="{path}"', "-o", str(lib), str(HERE / "kept_memory_host.cpp")], check=True)
    lib = ctypes.CDLL(str(lib))
    u64 = ctypes.c_uint64
    lib.fake_device.argtypes = [u64]
    lib.fake_used.restype = lib.fake_plain.restype = u64
    lib.block_alloc.argtypes, lib.block_alloc.restype = [u64, ctypes.POINTER(u64)], u64
    lib.block_free.argtypes = [u64, u64]
    lib.scratch.argtypes, lib.scratch.restype = [u64], u64
    lib.scratch_free.argtypes = [u64]
    lib.words.argtypes, lib.words.restype = [u64], u64
    return lib


@pytest.fixture
def device(request):
    lib = load(SOURCE, request.node.name.replace("[", "_").replace("]", ""))
    lib.fake_device(8 * GB)
    return lib


def block(device, size):
    got = ctypes.c_uint64()
    return device.block_alloc(size, ctypes.byref(got)), got.value


@pytest.mark.parametrize("end", [0, 1])
@pytest.mark.parametrize("other", [0, 1])
def test_a_build_goes_on_while_a_scene_ends(device, end, other):
    """A scene's end waits for the device; other threads do not wait for it."""
    assert device.runs_beside(end, other) == 1
    assert device.fake_used() == 0


def test_blocks_are_kept_and_given_back(device):
    device.begin()
    device.begin()
    p, got = block(device, GB // 2)
    device.block_free(p, got)
    assert device.fake_plain() == GB // 2  # kept
    assert block(device, GB // 2 - 100)[0] == p  # and used again, if it fits
    q, got_q = block(device, GB // 4)
    assert q != p and got_q == GB // 4
    device.block_free(p, got)
    device.block_free(q, got_q)
    assert device.fake_plain() == GB // 2 + GB // 4
    big, got_big = block(device, 8 * GB - GB // 4)  # all that is kept comes back for it
    assert big and got_big == 8 * GB - GB // 4
    device.block_free(big, got_big)  # too large to keep
    device.end()
    device.end()
    assert device.fake_used() == 0


def test_nothing_is_kept_for_a_lone_scene(device):
    device.begin()
    p, got = block(device, GB // 8)
    device.block_free(p, got)
    device.end()
    assert device.fake_used() == 0


def test_scratch_takes_what_is_kept(device):
    """A build whose keys fit only without a destroyed scene's pool, or without the
    scratch that it has itself freed, gets them."""
    device.begin()
    device.begin()
    p, got = block(device, GB)
    device.block_free(p, got)
    assert device.fake_used() == GB
    a = device.scratch(7 * GB + GB // 2)
    assert a and device.fake_used() == 7 * GB + GB // 2
    device.scratch_free(a)  # the stream has not come to it
    b = device.scratch(7 * GB + 3 * (GB // 4))
    assert b and device.fake_used() == 7 * GB + 3 * (GB // 4)
    device.scratch_free(b)
    assert not device.scratch(8 * GB + 1)  # more than there is
    assert device.fake_last_error() == 0  # nothing left for the next call to find
    device.end()
    device.end()
    assert device.fake_used() == 0


def test_any_allocation_takes_what_is_kept(device):
    device.begin()
    device.begin()
    p, got = block(device, GB)
    device.block_free(p, got)
    assert device.words((7 * GB + GB // 2) // 4)
    assert device.fake_used() == 7 * GB + GB // 2
    assert not device.words(GB // 4)
    assert device.fake_last_error() == 0


def test_every_allocation_of_the_library_can():
    """Device memory is asked for in kept_memory.cpp alone, which has what is kept
    given back where it does not fit.  (The ordering's scratch and the ray counter,
    small pieces of a stream-ordered pool, do without.)"""
    for f in sorted(SOURCE.parent.iterdir()):
        if f.suffix in (".cpp", ".cu", ".cuh", ".h") and f != SOURCE:
            for call in ("cudaMalloc(", "cudaMallocAsync(", "cudaMallocManaged(", "cudaMallocPitch("):
                assert call not in f.read_text(), f"{f.name}: {call}"
