"""What the passes derive from fields set as a list in device memory (for later stages run by hand) is what single calls
leave: also where a label or a mass of 0 in the list changes which derived values a particle has, and for velocities,
whose copy in the gather records is all that follows a sorted, aligned one."""

import ctypes

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu

LISTS = [("density", "label"), ("label", "saturation"), ("density", "mass", "pressure"), ("vel",), ("vel", "col"),
         ("voidage", "vel"), ("pressure", "label", "vel", "mass", "density"), ("mass", "label", "mass")]


@pytest.mark.parametrize("names", LISTS, ids="-".join)
@pytest.mark.parametrize("order", ["sorted", "id"])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("stages", [("sort", "density"), ("sort", "density", "avgflow", "voidage_adhesion")])
def test_derived_values_of_a_list(cuda_lib, names, order, offset, stages):
    torch = pytest.importorskip("torch")
    from sph_seepage_flows_gb300.capi import FIELDS, ORDER, Simulation
    sims = [Simulation(scenes.tiny(seed=9)) for _ in range(2)]
    n = sims[0].size()
    for sim in sims:
        sim.substeps_fixed(1e-4, 2)
        for st in stages:
            sim.stage(st, 1e-4)
    rng = np.random.default_rng(len(names))
    bufs = []
    for k in names:
        v = sims[0].field(k, order=order)
        if k == "label":
            v = np.where(rng.random(n) < 0.1, 1 - v, v).astype(np.int32)
        else:
            v = (v * rng.uniform(0.8, 1.2, v.shape)).astype(np.float32)
        if k == "mass":
            v[rng.random(n) < 0.05] = 0
        v = v.reshape(-1)
        t = torch.zeros(v.size + 4, dtype=torch.int32 if k == "label" else torch.float32, device="cuda")[offset:][:v.size]
        t.copy_(torch.from_numpy(v))
        bufs.append(t)
    torch.cuda.synchronize()
    lib, h = sims[0].lib, sims[0].h
    ids = (ctypes.c_int32 * len(names))(*[FIELDS[k][0] for k in names])
    ptr = (ctypes.c_void_p * len(names))(*[t.data_ptr() for t in bufs])
    assert lib.sf_set_fields(h, 0, len(names), ids, ORDER[order], ptr, n, 1) == 0
    for k, t in zip(names, bufs):
        assert lib.sf_set_field(sims[1].h, 0, FIELDS[k][0], ORDER[order], t.data_ptr(), n, 1) == 0
    for sim in sims:
        sim.stage("sand_momentum", 1e-4)
        sim.stage("water_momentum", 1e-4)
    for k in FIELDS:
        assert np.array_equal(sims[0].field(k), sims[1].field(k), equal_nan=True), k
