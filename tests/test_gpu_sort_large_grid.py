"""Few particles in a grid of a million cells: the passes over the cell table are shared by as many threads as the table
needs, not by those of the particles alone, in the sort and where the order is reset with counts in the table."""

import time

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(cells_per_side):
    h = scenes.tiny().params.sph_kernel_radius
    side = (cells_per_side + 0.25) * h
    sc = scenes.block_scene("wide", (side,) * 3, (5, 5, 5), (5, 5, 5), 0.02, 1)
    assert np.prod(sc.bparams.grid_size[:]) == cells_per_side ** 3
    sc.bpos, sc.blabel = sc.bpos[:0], sc.blabel[:0]
    return sc


def test_sort_in_a_large_grid_takes_no_multiple_of_one_in_a_small_grid(cuda_lib):
    from sph_seepage_flows_gb300.capi import Simulation
    best = {}
    for cells in (20, 100):
        sim = Simulation(_scene(cells))
        for _ in range(5):
            sim.stage("sort")
            sim.synchronize()
            t = time.perf_counter()
            for _ in range(50):
                sim.stage("sort")
            sim.synchronize()
            best[cells] = min(best.get(cells, 1.0), (time.perf_counter() - t) / 50)
    # the passes over the table take some 5 us more; with the blocks of the particles alone it was 65 times as long
    assert best[100] < 10 * best[20], best


def test_order_reset_with_counts_in_a_large_grid(cuda_lib):
    from sph_seepage_flows_gb300.capi import Simulation
    sc = _scene(100)
    outs = []
    for again in (False, True):
        sim = Simulation(sc)
        if again:
            sim.substeps_fixed(1e-4, 3)  # leaves counts in the table
            sim.reset_order()
            assert np.array_equal(sim.field("id"), np.arange(sc.n))
            sim.set_fields({"pos": sc.pos, "vel": sc.vel}, order="id")
        sim.substeps_fixed(1e-4, 2)
        outs.append({k: sim.field(k) for k in ("id", "key", "pos", "vel")} | {"table": sim.cell_table(0)})
    for k, v in outs[0].items():
        assert np.array_equal(v, outs[1][k]), k
