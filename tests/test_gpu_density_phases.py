"""The one-lane density pass tests candidates two to an instruction from even
slots on, 32 to a chunk, keeps the chunks' hit masks and takes the hits
afterwards, merging water and boundary neighbours by the end of their cells.
Checked bit for bit against the FP32 oracle where that can go wrong: columns
of fewer and more than 32 candidates, more chunks than are kept, odd starts,
walls on three sides, and more boundary neighbours than the boundary list
holds."""

import numpy as np
import pytest

from helpers import compare_stages
from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu

T_FRAME = 1.0 / 30.0
TOL = 1e-5   # as tests/test_gpu_parity.py, for the fields through powf and the adhesion spline


def corner_scene(squeeze, shape_points):
    """Sand and water lattices of odd sizes in the low corner of the box, both
    drawn towards the corner (squeeze times the pitch), and a patch of shape
    boundary particles at the floor."""
    sc = scenes.block_scene("corner", (0.4, 0.4, 0.4), (5, 7, 9), (7, 5, 11), 0.02, 3,
                            sand_origin=(0.05, 0.021, 0.023), water_origin=(0.021, 0.02, 0.025))
    sc.pos[:] = (0.02 + (sc.pos - np.float32(0.02)) * np.float32(squeeze)).astype(np.float32)
    rng = np.random.default_rng(8)
    return scenes.add_shape_boundary(sc, rng.uniform(0.0, 0.06, (shape_points, 3)).astype(np.float32)
                                     * np.float32([1.0, 0.2, 1.0]))


@pytest.mark.parametrize("squeeze, shape_points", [(1.0, 0), (0.8, 0), (0.55, 0), (0.4, 0), (1.0, 300)])
def test_one_lane_density_matches_the_oracle(cuda_lib, oracle_mod, squeeze, shape_points):
    from sph_seepage_flows_gb300.capi import Simulation
    sc = corner_scene(squeeze, shape_points)
    sim = Simulation(sc)
    sim.set_lanes(1)
    o32 = oracle_mod.Oracle(sc, 32)
    compare_stages(sim, o32, T_FRAME, True, TOL, stages=["sort", "density", "avgflow", "voidage_adhesion"])
    assert sim.check_error() == 0


def test_density_after_positions_set_between_stages(cuda_lib, oracle_mod):
    """Positions written after the sort reach the density pass (its slot-pair copies follow)."""
    from sph_seepage_flows_gb300.capi import Simulation
    sc = corner_scene(0.8, 0)
    sim = Simulation(sc)
    sim.set_lanes(1)
    o32 = oracle_mod.Oracle(sc, 32)
    sim.stage("sort", T_FRAME)
    o32.stage("sort", T_FRAME, adaptive=False)
    pos = (sim.field("pos") + np.random.default_rng(4).uniform(-2e-4, 2e-4, (sc.n, 3))).astype(np.float32)
    sim.set_field("pos", pos)
    o32.set_field("pos", pos)
    compare_stages(sim, o32, T_FRAME, True, TOL, stages=["density"])


@pytest.mark.parametrize("lanes", [1, 2, 8])
def test_sand_volume_of_the_chained_passes(cuda_lib, lanes):
    """In a whole substep the density pass sums the sand volume around sand; run stage by stage the average-flow pass
    does. Both give the same bits, with sand of several masses and lists that overflow too."""
    from sph_seepage_flows_gb300.capi import Simulation
    for squeeze in (0.8, 0.3):
        sc = corner_scene(squeeze, 0)
        sand = sc.label == 1
        sc.mass[sand] *= np.float32([1.0, 0.7, 1.3])[np.arange(int(sand.sum())) % 3]
        whole, staged = Simulation(sc), Simulation(sc)
        for sim in (whole, staged):
            sim.set_lanes(lanes)
        whole.substeps_fixed(1e-5, 1)
        for st in ("sort", "density", "avgflow", "voidage_adhesion", "sand_momentum", "water_momentum", "integrate"):
            staged.stage(st, 1e-5)
        for name in ("id", "density", "voidage", "saturation", "avg_flow", "acc", "vel", "pos"):
            assert np.array_equal(whole.field(name), staged.field(name), equal_nan=True), (squeeze, name)
