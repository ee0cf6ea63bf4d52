"""The descent that lanes leave and take up again (libsvo_b200/csrc/traverse.cuh,
stream_rays_kernel), compiled for the host: a call ends its ray or moves it on by
a pass, even where a lane finds itself alone before the first one, and the records
are the oracle's however often a ray was left."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle
from rays import edge_rays, random_octree_pool

HERE = Path(__file__).resolve().parent / "hostsim"
LIB = HERE / "_build" / "libyield_host.so"


@pytest.fixture(scope="module")
def lib():
    src = HERE / "yield_host.cpp"
    deps = [src, HERE / "host_shim.h", HERE.parent.parent / "libsvo_b200" / "csrc" / "traverse.cuh"]
    if not LIB.is_file() or any(LIB.stat().st_mtime < d.stat().st_mtime for d in deps):
        LIB.parent.mkdir(parents=True, exist_ok=True)
        subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-fast-math", "-fPIC", "-shared",
                        "-o", str(LIB), str(src)], check=True)
    lib = ctypes.CDLL(str(LIB))
    vp = ctypes.c_void_p
    lib.host_cast_yielding.argtypes = [vp, ctypes.c_uint64, vp, vp, ctypes.c_uint64, ctypes.c_float, ctypes.c_int,
                                       ctypes.c_int, ctypes.c_int, vp, vp]
    lib.host_cast_yielding.restype = ctypes.c_uint64
    return lib


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("keep", [0, 1, 20])
def test_every_call_moves_its_ray_on(lib, keep, flat):
    nodes, _ = random_octree_pool(keep, depth=6, fill=0.3)
    nodes = nodes.copy()
    if flat:
        nodes[:, 0] += np.arange(len(nodes), dtype=np.uint32)
    o, d = edge_rays(n_random=4000, seed=keep)
    S = 6 if flat else 13
    o, d = np.ascontiguousarray(o, dtype=np.float32), np.ascontiguousarray(d, dtype=np.float32)
    got = np.zeros(len(o), dtype=oracle.HIT_DTYPE)
    calls = ctypes.c_uint32()
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (nodes, o, d, got)]
    idle = lib.host_cast_yielding(p[0], len(nodes), p[1], p[2], len(o), 0.001, S, int(flat), keep, p[3],
                                  ctypes.byref(calls))
    assert idle == 0
    assert calls.value == 1 if keep == 0 else calls.value > 20
    want, _ = oracle.cast_rays(nodes, o, d, 0.001, flat=flat, stack_size=S)
    for k in ("node", "depth", "hit", "flags", "loops", "fetches"):
        assert np.array_equal(got[k], want[k]), k
    assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
