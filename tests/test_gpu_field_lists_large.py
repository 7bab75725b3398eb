"""Field lists in device memory of a scene above the sizes up to which one launch moves the whole list: the values are
those of calls of their own, in both orders, with buffers off the 16-byte grid among them, and a list takes no longer
than those calls."""

import ctypes
import time

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu

NAMES = ("pos", "density", "vel", "max_saturation", "col", "cda0asat", "amcamcp", "pressure", "mass")


@pytest.fixture(scope="module")
def large(cuda_lib):
    from sph_seepage_flows_gb300.capi import Simulation
    sc = scenes.block_scene("fields", (9.0,) * 3, (2, 2, 2), (2, 2, 2), 0.02, 1)
    n = 2_000_003
    rng = np.random.default_rng(0)
    pick = rng.integers(0, sc.n, n)
    for name in ("vel", "col", "label", "mass", "radius", "cda0asat", "amcamcp"):
        setattr(sc, name, getattr(sc, name)[pick])
    sc.pos = rng.uniform(0.1, 8.9, (n, 3)).astype(np.float32)
    sim = Simulation(sc)
    sim.stage("sort")
    sim.synchronize()
    return sim


def _call(sim, fn, names, bufs, order):
    from sph_seepage_flows_gb300.capi import FIELDS, ORDER
    ids = (ctypes.c_int32 * len(names))(*[FIELDS[k][0] for k in names])
    ptr = (ctypes.c_void_p * len(names))(*[b.data_ptr() for b in bufs])
    sim._check(getattr(sim.lib, fn)(sim.h, 0, len(names), ids, ORDER[order], ptr, sim.size(0), 1))


@pytest.mark.parametrize("order", ["sorted", "id"])
@pytest.mark.parametrize("offset", [0, 1])
def test_large_list_equals_single_calls(large, order, offset):
    torch = pytest.importorskip("torch")
    from sph_seepage_flows_gb300.capi import FIELDS
    sim, n = large, large.size(0)
    gen = torch.Generator("cuda").manual_seed(offset)
    make = lambda k: torch.rand(n * FIELDS[k][1] + 4, device="cuda", generator=gen)[offset:][:n * FIELDS[k][1]]  # noqa: E731
    values = [make(k) for k in NAMES]
    reads = {}
    for single in (True, False):
        # from the same state
        start = [torch.full((n * FIELDS[k][1],), 0.5, device="cuda") for k in NAMES]
        torch.cuda.synchronize()
        _call(sim, "sf_set_fields", NAMES, start, "sorted")
        for part in ([(k,) for k in NAMES] if single else [NAMES]):
            _call(sim, "sf_set_fields", part, [values[NAMES.index(k)] for k in part], order)
        got = [make(k) for k in NAMES]
        torch.cuda.synchronize()
        for part in ([(k,) for k in NAMES] if single else [NAMES]):
            _call(sim, "sf_get_fields", part, [got[NAMES.index(k)] for k in part], order)
        sim.synchronize()
        reads[single] = got
    for k, v, a, b in zip(NAMES, values, reads[True], reads[False]):
        assert torch.equal(a, v), k
        assert torch.equal(b, v), k


def test_large_list_takes_no_longer_than_single_calls(large):
    torch = pytest.importorskip("torch")
    from sph_seepage_flows_gb300.capi import FIELDS, ORDER
    sim, n, names = large, large.size(0), ("pos", "vel")
    bufs = [torch.full((n * 3,), 0.5, device="cuda") for _ in names]
    torch.cuda.synchronize()

    def single():
        for k, b in zip(names, bufs):
            sim._check(sim.lib.sf_set_field(sim.h, 0, FIELDS[k][0], ORDER["sorted"], b.data_ptr(), n, 1))

    best = {}
    for _ in range(7):
        for what, fn in (("single", single), ("list", lambda: _call(sim, "sf_set_fields", names, bufs, "sorted"))):
            fn()
            sim.synchronize()
            t = time.perf_counter()
            for _ in range(100):
                fn()
            sim.synchronize()
            best[what] = min(best.get(what, 1.0), (time.perf_counter() - t) / 100)
    assert best["list"] < 1.15 * best["single"], best
