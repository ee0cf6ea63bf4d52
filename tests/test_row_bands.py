"""The launches of a frame taller than one grid (libsvo_b200/csrc/row_bands.h): every
row once, at heights up to the largest that is accepted."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent / "hostsim"
GRID = 65535
LARGEST = 0xFFFFFFF0


@pytest.fixture(scope="module")
def lib():
    out = HERE / "_build" / "librow_bands.so"
    out.parent.mkdir(parents=True, exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-o", str(out), str(HERE / "row_bands_host.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(out))
    lib.bands.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_int64]
    lib.bands.restype = ctypes.c_int64
    return lib


@pytest.mark.parametrize("block_h", [1, 2, 4, 8])
@pytest.mark.parametrize("height", [1, 7, 8, 9, 65535, 65536, 524280, 524281, 4294901760, 4294901761, LARGEST])
def test_every_row_is_in_one_band(lib, height, block_h):
    cap = 70000
    out = np.zeros((cap, 3), dtype=np.uint32)
    n = lib.bands(height, block_h, out.ctypes.data_as(ctypes.c_void_p), cap)
    assert n == -(-height // (GRID * block_h))
    b = out[:n].astype(np.int64)
    assert b[0, 0] == 0 and (b[1:, 0] == b[:-1, 0] + b[:-1, 1]).all() and b[-1, 0] + b[-1, 1] == height
    assert (b[:, 2] == -(-b[:, 1] // block_h)).all() and (b[:, 2] <= GRID).all()
