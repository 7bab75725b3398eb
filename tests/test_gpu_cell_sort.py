"""The sort stage is the stable order of the cell keys, whichever of its two
forms runs: the counting sort, or the radix sort where the grid has many more
cells than the handle has slots. Checked against numpy's stable argsort:
shuffled creation order, spare capacity (parked slots), one crowded cell,
several scenes in one handle, sizes at the edges of blocks and table tiles,
and repeated sorts after the particles moved."""

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu


def make_scene(n, side, seed, crowd=0):
    """n particles in random order and places of a cube; the first `crowd` of them in one cell."""
    sc = scenes.block_scene("sort", (side,) * 3, (2, 2, 2), (2, 2, 2), 0.02, seed)
    rng = np.random.default_rng(seed)
    pick = rng.integers(0, sc.n, n)
    for name in ("vel", "col", "label", "mass", "radius", "cda0asat", "amcamcp"):
        setattr(sc, name, getattr(sc, name)[pick])
    sc.pos = rng.uniform(0.0, side, (n, 3)).astype(np.float32)
    sc.pos[:crowd] = (0.5 * side + rng.uniform(0.0, 1e-3, (crowd, 3))).astype(np.float32)
    return sc


def keys_of(sc, pos):
    b = sc.bparams
    g = np.array(b.grid_size[:])
    q = (pos - np.float32(b.lowest_point[:])) / np.float32(b.kernel_radius)
    c = np.minimum(np.maximum(q.astype(np.int64), 0), g - 1)
    return (c[:, 0] * g[1] + c[:, 1]) * g[2] + c[:, 2], int(g.prod())


@pytest.mark.parametrize("sizes, side, spare, crowd", [
    ((1,), 0.4, 0, 0), ((255, 256, 257), 0.4, 0, 0), ((1000,), 0.4, 5000, 0), ((3000, 40), 0.3, 700, 2500),
    ((20011,), 1.3, 0, 0), ((1500,), 6.0, 300, 0)])
def test_sort_is_the_stable_key_order(cuda_lib, sizes, side, spare, crowd):
    from sph_seepage_flows_gb300.capi import Simulation
    scs = [make_scene(n, side, 10 + k, min(crowd, n)) for k, n in enumerate(sizes)]
    sim = Simulation(scs, capacity=[sc.n + spare for sc in scs])
    order = [np.arange(sc.n) for sc in scs]   # ids in slot order
    pos = [sc.pos for sc in scs]              # by id
    rng = np.random.default_rng(1)
    for turn in range(3):
        sim.stage("sort")
        for s, sc in enumerate(scs):
            keys, cells = keys_of(sc, pos[s])
            order[s] = order[s][np.argsort(keys[order[s]], kind="stable")]
            assert np.array_equal(sim.field("id", scene=s), order[s]), (turn, s)
            assert np.array_equal(sim.field("key", scene=s), keys[order[s]]), (turn, s)
            assert np.array_equal(sim.field("pos", scene=s), pos[s][order[s]]), (turn, s)
            assert np.array_equal(sim.field("mass", scene=s), sc.mass[order[s]]), (turn, s)
            table = np.searchsorted(keys[order[s]], np.arange(cells + 1))
            assert np.array_equal(sim.cell_table(0, scene=s), table), (turn, s)
            # some particles to other places, a few out of the grid
            move = rng.random(sc.n) < 0.2
            pos[s] = pos[s].copy()
            pos[s][move] = rng.uniform(-0.05, side + 0.05, (int(move.sum()), 3)).astype(np.float32)
            sim.set_field("pos", pos[s], order="id", scene=s)
    assert sim.check_error() == 0
