"""When a position that is not finite is reported (sf_check_error): by the sort that meets it, in both forms of the sort
stage, and not by the substep that wrote it, since the caller may replace the position in between."""

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [0.4, 6.0])
@pytest.mark.parametrize("repaired", [True, False])
def test_a_position_out_of_range_is_reported_by_the_sort_that_meets_it(cuda_lib, side, repaired):
    from sph_seepage_flows_gb300.capi import Simulation
    sc = scenes.block_scene("far", (side,) * 3, (3, 3, 3), (3, 3, 3), 0.02, 3)
    lone = int(np.argmax(sc.label == 1))  # sand, which is not clamped to the box, without neighbours
    sc.pos[lone] = 0.3
    sim = Simulation(sc)
    good, still = sim.field("pos", order="id"), sim.field("vel", order="id")
    fast = still.copy()
    fast[lone] = 3e38
    for _ in range(2):
        sim.set_fields({"pos": good, "vel": fast}, order="id")
        sim.substeps_fixed(10.0, 1)
        assert not np.isfinite(sim.field("pos", order="id")[lone]).any()
        assert sim.check_error() == 0
        if repaired:
            sim.set_fields({"pos": good, "vel": still}, order="id")
        sim.stage("sort")
        assert sim.check_error() == (0 if repaired else 1)
