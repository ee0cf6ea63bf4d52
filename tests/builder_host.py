"""tests/hostsim/builder_host.cpp, built and bound."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent.parent
SRC = ROOT / "tests" / "hostsim" / "builder_host.cpp"
LIB = ROOT / "tests" / "hostsim" / "_build" / "libbuilder_host.so"


def load():
    csrc = ROOT / "libsvo_b200" / "csrc"
    deps = [SRC, csrc / "scene.cpp", csrc / "scene.h", csrc / "chunk_plan.h"]
    if not LIB.is_file() or any(LIB.stat().st_mtime < d.stat().st_mtime for d in deps):
        LIB.parent.mkdir(parents=True, exist_ok=True)
        subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-pthread", "-o", str(LIB), str(SRC)],
                       check=True)
    lib = ctypes.CDLL(str(LIB))
    vp, u64, u32 = ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint32
    lib.plan.argtypes, lib.plan.restype = [vp, u64, u32, u32, u64, u64, vp, u64], ctypes.c_int64
    lib.near_voxels.argtypes, lib.near_voxels.restype = [vp, u32, ctypes.c_int, vp, u64], u64
    return lib


def near_voxels(lib, triangle, depth, margin=3):
    """The sorted codes of the voxels that a triangle long in x overlaps."""
    t = np.ascontiguousarray(triangle, dtype=np.float32).reshape(9)
    p = t.ctypes.data_as(ctypes.c_void_p)
    n = lib.near_voxels(p, depth, margin, None, 0)
    codes = np.zeros(n, dtype=np.uint64)
    lib.near_voxels(p, depth, margin, codes.ctypes.data_as(ctypes.c_void_p), n)
    return np.sort(codes)


def leaves(nodes, depth):
    """The sorted leaf codes of a pool of one treelet holding a whole octree, and the
    leaves' records."""
    first, masks = nodes[:, 0].astype(np.int64), nodes[:, 1]
    at, code = np.zeros(1, dtype=np.int64), np.zeros(1, dtype=np.uint64)
    for _ in range(depth):
        valid = (masks[at] >> 8) & 0xFF
        before = np.zeros(len(at), dtype=np.int64)
        nxt, codes = [], []
        for c in range(8):
            has = (valid >> c) & 1 == 1
            nxt.append(at[has] + first[at[has]] + before[has])
            codes.append((code[has] << np.uint64(3)) | np.uint64(c))
            before += has
        at, code = np.concatenate(nxt), np.concatenate(codes)
    order = np.argsort(code)
    return code[order], at[order]


def sliver(corner, length, depth, rng):
    """A triangle of `length` along x and nearly as long along y and z, about a
    voxel wide: its box has far more columns than it overlaps voxels."""
    voxel = 0.5 ** depth
    a = np.asarray(corner, dtype=np.float64) + rng.uniform(0, voxel, 3)
    b = a + length * np.array([1.0, 0.93, 0.81])
    c = a + voxel * np.array([0.0, 1.1, -0.4])
    return np.stack([a, b, c]).astype(np.float32)
