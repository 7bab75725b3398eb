"""A whole substep's passes up to voidage / adhesion give the same bits for every lane count and for the pairings of the
density's and the average flow's that the automatic choice makes (by the slots of a handle, which spare capacity counts
among): the sand volume that the density pass sums reaches the average flow of any lane count. With shape boundaries,
sand of several masses, lists that overflow and more boundary neighbours than the boundary list holds."""

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes
from test_gpu_density_phases import corner_scene

pytestmark = pytest.mark.gpu

FIELDS = ("id", "neighbors", "density", "pressure", "voidage", "saturation", "max_saturation", "col", "avg_flow")


def _fields(sc, lanes, slots, by_stages):
    from sph_seepage_flows_gb300.capi import Simulation
    sim = Simulation(sc, capacity=max(slots, sc.n))
    if lanes:
        sim.set_lanes(lanes)
    if by_stages:
        for st in ("sort", "density", "avgflow", "voidage_adhesion", "sand_momentum", "water_momentum", "integrate"):
            sim.stage(st, 1e-5)
    else:
        sim.substeps_fixed(1e-5, 1)
    out = {k: sim.field(k) for k in FIELDS}
    assert sim.check_error() == 0
    sim.close()
    return out


@pytest.mark.parametrize("squeeze, shape_points", [(1.0, 0), (0.8, 300), (0.3, 0)])
@pytest.mark.parametrize("lanes, slots", [
    (2, 0), (4, 0), (8, 0),
    (0, 0),        # density and average flow with 8 lanes each
    (0, 40_000),   # 4 and 4
    (0, 200_000),  # 1 (loading ahead) and 2
    (0, 650_000),  # 1 and 1
])
def test_lane_counts_and_pairings_give_the_same_bits(cuda_lib, squeeze, shape_points, lanes, slots):
    sc = corner_scene(squeeze, shape_points)
    sand = sc.label == 1
    sc.mass[sand] *= np.float32([1.0, 0.7, 1.3])[np.arange(int(sand.sum())) % 3]
    want = _fields(sc, 1, 0, by_stages=True)
    for by_stages in (False, True):
        got = _fields(sc, lanes, slots, by_stages)
        for k, v in want.items():
            assert np.array_equal(got[k], v, equal_nan=True), (k, by_stages)
