"""Stages run by hand over states that whole substeps do not pass through: particles parked without a sort in between
(a parked sand particle keeps its sign, -0) and labels changed before a density pass alone. Every form of the density
pass leaves the same lists and the same values for the stages after it."""

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu

FORMS = [(1, 0, False), (1, 0, True), (1, 700_000, False), (2, 0, False), (4, 0, False), (8, 0, False)]


def _form(sc, lanes, slots, staged):
    from sph_seepage_flows_gb300.capi import Simulation
    sim = Simulation(sc, capacity=max(slots, sc.n))
    sim.set_lanes(lanes)
    sim.set_density_staging(staged)
    return sim


@pytest.mark.parametrize("stages", [("sand_momentum", "water_momentum"), ("avgflow", "voidage_adhesion", "water_momentum")])
def test_density_after_particles_were_parked(cuda_lib, stages):
    want = None
    for lanes, slots, staged in FORMS:
        sc = scenes.tiny(seed=4)
        sim = _form(sc, lanes, slots, staged)
        for st in ("sort", "density", "avgflow", "voidage_adhesion"):
            sim.stage(st, 1e-4)
        sim.set_lanes(1)  # the momentum sums of every form in one order
        sim.stage("sand_momentum", 1e-4)
        mass = sim.field("mass", order="id")
        mass[np.random.default_rng(0).random(sc.n) < 0.2] = 0
        sim.set_field("mass", mass, order="id")
        sim.set_lanes(lanes)
        sim.stage("density", 1e-4)
        sim.set_lanes(1)
        for st in stages:
            sim.stage(st, 1e-4)
        got = {k: sim.field(k) for k in ("id", "neighbors", "density", "voidage", "saturation", "acc")}
        want = want or got
        for k, v in want.items():
            assert np.array_equal(got[k], v, equal_nan=True), (k, lanes, slots, staged)


def test_voidage_after_a_density_pass_alone(cuda_lib):
    """A density pass by itself does not touch what the average flow left: labels changed before and after it."""
    want = None
    for lanes, slots, staged in FORMS:
        sc = scenes.tiny(seed=4)
        sim = _form(sc, lanes, slots, staged)
        sim.stage("sort")
        rng = np.random.default_rng(1)
        for _ in range(2):
            sim.stage("density", 1e-4)
            label = sim.field("label", order="id")
            sim.set_field("label", np.where(rng.random(sc.n) < 0.3, 1 - label, label).astype(np.int32), order="id")
        sim.stage("sort")
        sim.stage("density", 1e-4)
        sim.stage("voidage_adhesion", 1e-4)
        got = {k: sim.field(k) for k in ("id", "neighbors", "density", "voidage", "adhesion")}
        want = want or got
        for k, v in want.items():
            assert np.array_equal(got[k], v, equal_nan=True), (k, lanes, slots, staged)
