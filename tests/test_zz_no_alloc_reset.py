"""sf_cell_sort_noalloc after cudaDeviceReset, in a process of its own: the call works whatever took the old addresses
by then (the library's module loaded again by another call, other allocations on the device and pinned on the host),
and a position that is not finite is still reported."""

import glob
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, sys
import numpy as np
from sph_seepage_flows_gb300 import capi, scenes

between, rt = sys.argv[1], ctypes.CDLL(sys.argv[2])
lib = capi.load()
sc = scenes.tiny()
b = sc.bparams
cells = int(np.prod(b.grid_size[:]))
c = ((sc.pos - np.float32(b.lowest_point[:])) / np.float32(b.kernel_radius)).astype(np.int64)
c = np.clip(c, 0, np.array(b.grid_size[:]) - 1)
keys = (c[:, 0] * b.grid_size[1] + c[:, 1]) * b.grid_size[2] + c[:, 2]
want = np.argsort(keys, kind="stable")
table = np.searchsorted(keys[want], np.arange(cells + 1))

def ok(status):
    assert status == 0, status

def alloc(nbytes):
    p = ctypes.c_void_p()
    ok(rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(nbytes)))
    return p

def host(nbytes):
    p = ctypes.c_void_p()
    ok(rt.cudaHostAlloc(ctypes.byref(p), ctypes.c_size_t(nbytes), 0))
    ctypes.memset(p, 0x55, nbytes)
    return p

def sort(pos):
    pos = np.ascontiguousarray(pos, np.float32)
    perm, cs = np.full(sc.n, -1, np.int32), np.full(cells + 1, -1, np.int32)
    bufs = [alloc(a.nbytes) for a in (pos, perm, cs)]
    ok(rt.cudaMemcpy(bufs[0], ctypes.c_void_p(pos.ctypes.data), ctypes.c_size_t(pos.nbytes), 1))
    st = lib.sf_cell_sort_noalloc(ctypes.byref(b), bufs[0], sc.n, bufs[1], bufs[2], None)
    for a, d in ((perm, bufs[1]), (cs, bufs[2])):
        ok(rt.cudaMemcpy(ctypes.c_void_p(a.ctypes.data), d, ctypes.c_size_t(a.nbytes), 2))
    for d in bufs:
        ok(rt.cudaFree(d))
    return st, perm, cs

bad = sc.pos.copy()
bad[7, 1] = np.nan
for life in range(3):
    if life:
        ok(rt.cudaDeviceReset())
    if between == "module":
        sim = capi.Simulation(sc)
        sim.substeps_fixed(1e-4, 2)
        sim.synchronize()
        sim.close()
    pinned = [host(64 << k) for k in range(12) for _ in range(4)] if between == "buffers" else []
    held = [alloc(5 << 20) for _ in range(40)] if between == "buffers" else []
    for _ in range(2):
        st, perm, cs = sort(sc.pos)
        assert st == 0, lib.sf_last_error_string(None)
        assert np.array_equal(perm, want) and np.array_equal(cs, table), (between, life)
        assert sort(bad)[0] == 4, (between, life)
    for k, p in enumerate(pinned):
        size = 64 << (k // 4)
        assert ctypes.string_at(p, size) == b"\x55" * size, (between, life, k)
print("reset ok")
"""


@pytest.mark.parametrize("between", ["nothing", "module", "buffers"])
def test_noalloc_sort_after_reset(cuda_lib, between):
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    found = sorted(glob.glob(os.path.join(home, "lib64", "libcudart.so*")))
    if not found:
        pytest.skip("no shared CUDA runtime to reset the device with")
    r = subprocess.run([sys.executable, "-c", CHILD, between, found[0]], cwd=ROOT, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and "reset ok" in r.stdout, r.stdout + r.stderr
