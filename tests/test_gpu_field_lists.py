"""Several fields in device memory move in one launch (sf_get_fields /
sf_set_fields): the same values as one call per field, in both orders, for
more fields than a launch takes, fields named twice, boundary fields among
them and an invalid field at the end; and sf_reset_order over scenes of
uneven sizes with spare capacity."""

import ctypes

import numpy as np
import pytest
import torch

from sph_seepage_flows_gb300 import scenes
from sph_seepage_flows_gb300.params import BFIELDS, FIELDS

pytestmark = pytest.mark.gpu


def call(sim, fn, scene, names, order, tensors, n):
    ids = (ctypes.c_int32 * len(names))(*[(FIELDS.get(k) or BFIELDS[k])[0] if isinstance(k, str) else k for k in names])
    ptrs = (ctypes.c_void_p * len(names))(*[t.data_ptr() for t in tensors])
    return fn(sim.h, scene, len(names), ids, order, ptrs, n, 1)


def prepared():
    from sph_seepage_flows_gb300.capi import Simulation
    scs = [scenes.tiny(seed=3), scenes.tiny(seed=4, sand=(5, 3, 7), water=(3, 9, 4))]
    sim = Simulation(scs, capacity=[scs[0].n + 300, scs[1].n])
    sim.substeps_fixed(1e-4, 3)
    return scs, sim


@pytest.mark.parametrize("order", ["sorted", "id"])
def test_fields_in_one_launch_equal_single_calls(cuda_lib, order):
    scs, sim = prepared()
    code = {"sorted": 0, "id": 1}[order]
    names = list(FIELDS) + ["vel", "pos"]
    for s, sc in enumerate(scs):
        out = [torch.zeros(sc.n * FIELDS[k][1], dtype=torch.int32 if FIELDS[k][2] == np.int32 else torch.float32,
                           device="cuda") for k in names]
        assert call(sim, sim.lib.sf_get_fields, s, names, code, out, sc.n) == 0
        sim.synchronize()
        for k, t in zip(names, out):
            assert np.array_equal(t.cpu().numpy(), sim.field(k, order=order, scene=s).reshape(-1), equal_nan=True), k
        # set: a list (one field twice: the last one counts) against single calls
        rng = np.random.default_rng(s)
        new = {k: sim.field(k, order=order, scene=s) for k in ("vel", "mass", "saturation", "voidage", "col", "acc")}
        new = {k: (v * rng.uniform(0.9, 1.1, v.shape)).astype(np.float32) for k, v in new.items()}
        for k, v in new.items():
            sim.set_field(k, v, order=order, scene=s)
        state = {k: sim.field(k, scene=s) for k in FIELDS}
        dev = {k: torch.from_numpy(v).cuda() for k, v in new.items()}
        names2 = ["acc"] + list(new)
        src = [torch.zeros_like(dev["acc"])] + [dev[k] for k in new]
        torch.cuda.synchronize()
        assert call(sim, sim.lib.sf_set_fields, s, names2, code, src, sc.n) == 0
        for k in FIELDS:
            assert np.array_equal(sim.field(k, scene=s), state[k], equal_nan=True), k
        # an unknown field fails after the ones before it
        vel = torch.from_numpy(new["vel"] * 2).cuda()
        torch.cuda.synchronize()
        assert call(sim, sim.lib.sf_set_fields, s, ["vel", 99], code, [vel, vel], sc.n) == 1
        assert np.array_equal(sim.field("vel", order=order, scene=s), new["vel"] * 2)
        b = torch.zeros(sc.nb * 3, device="cuda")
        assert call(sim, sim.lib.sf_get_fields, s, ["bpos"], code, [b], sc.nb) == 0
        sim.synchronize()
        assert np.array_equal(b.cpu().numpy(), sim.field("bpos", scene=s).reshape(-1))


def test_reset_order_of_uneven_scenes(cuda_lib):
    scs, sim = prepared()
    before = [{k: sim.field(k, order="id", scene=s) for k in ("pos", "vel", "mass", "col", "radius")} for s in (0, 1)]
    sim.reset_order()
    for s, sc in enumerate(scs):
        assert np.array_equal(sim.field("id", scene=s), np.arange(sc.n))
        for k, v in before[s].items():
            assert np.array_equal(sim.field(k, scene=s), v), k
