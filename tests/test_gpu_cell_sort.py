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


@pytest.mark.parametrize("n, grid, crowd", [
    (1, (3, 3, 3), 0), (31, (1, 1, 1), 0), (33, (20, 10, 30), 33), (1025, (16, 8, 8), 256), (1025, (16, 8, 8), 257),
    (5000, (1, 1, 1), 0), (262144, (64, 50, 61), 0), (4099, (150, 100, 90), 0)])
def test_noalloc_sort_is_the_stable_key_order(cuda_lib, n, grid, crowd):
    """Both forms of the allocation-free sort: cells up to and above the size that the counting form orders, one cell for
    everything, tables of one tile, of many and with more cells than the counting form takes."""
    torch = pytest.importorskip("torch")
    import ctypes
    from sph_seepage_flows_gb300.params import boundary_params
    h = 0.04
    b = boundary_params((0.1, -0.2, 0.0), [0.1 + grid[0] * h + 0.01, -0.2 + grid[1] * h + 0.01, grid[2] * h + 0.01], h)
    assert list(b.grid_size[:]) == list(grid)
    rng = np.random.default_rng(n)
    lo = np.float32([0.1, -0.2, 0.0])
    pos = (lo + rng.uniform(-0.05, 1.05, (n, 3)) * np.float32(grid) * h).astype(np.float32)
    pos[rng.permutation(n)[:crowd]] = lo + np.float32(0.5 * h)
    q = ((pos - lo) / np.float32(h)).astype(np.int64)
    c = np.minimum(np.maximum(q, 0), np.array(grid) - 1)
    keys = (c[:, 0] * grid[1] + c[:, 1]) * grid[2] + c[:, 2]
    cells = int(np.prod(grid))
    want = np.argsort(keys, kind="stable")
    dpos = torch.from_numpy(pos).cuda()
    # the table at an odd word: it has no alignment beyond its elements'
    room = torch.full((cells + 3,), -7, dtype=torch.int32, device="cuda")
    table, perm = room[1:-1], torch.full((n,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        assert cuda_lib.sf_cell_sort_noalloc(ctypes.byref(b), dpos.data_ptr(), n, perm.data_ptr(), table.data_ptr(),
                                             None) == 0
        assert np.array_equal(perm.cpu().numpy(), want)
        assert np.array_equal(table.cpu().numpy(), np.searchsorted(keys[want], np.arange(cells + 1)))
        assert int(room[0]) == int(room[-1]) == -7


def test_counts_of_the_integrator_follow_what_happens_between_substeps(cuda_lib):
    """The integrator counts the positions it writes for the next sort. Whatever comes between (fields set, particles
    added, the order reset, stages by hand, an adjoint run), a run equals one whose every substep sorts from scratch."""
    from sph_seepage_flows_gb300.capi import Simulation
    dt = 1e-4

    def scenario(sim, n, substep):
        rng = np.random.default_rng(3)
        substep(2)
        pos = sim.field("pos", order="id")
        sim.set_field("pos", (pos + rng.uniform(-1e-3, 1e-3, pos.shape)).astype(np.float32), order="id")
        substep(3)
        sim.set_field("vel", sim.field("vel") * np.float32(0.5))
        substep(1)
        sim.add_sph_particles(rng.uniform(0.1, 0.3, (40, 3)), [0, 0, 1], [0, 0, 0], float(sim.scenes[0].params.sph_mass), 0.01)
        substep(2)
        sim.stage("sort")
        sim.stage("sort")
        substep(1)
        sim.stage("integrate", 1e-6)
        sim.stage("integrate", 1e-6)
        substep(1)
        sim.adjoint(dt, 3, sim.field("pos", order="id"), checkpoint_every=2)
        substep(2)
        sim.reset_order()
        substep(1)
        sim.step(1.0 / 30.0)
        sim.step(1.0 / 30.0)
        return {k: sim.field(k) for k in ("id", "key", "pos", "vel", "density", "acc")}, sim.cell_table(0)

    outs = []
    for by_hand in (False, True):
        sc = scenes.tiny(seed=5)
        sim = Simulation(sc, capacity=sc.n + 100)

        def substep(k):
            if not by_hand:
                sim.substeps_fixed(dt, k)
                return
            for _ in range(k):
                # a write of the positions as they are: the next sort counts anew
                sim.set_field("pos", sim.field("pos"))
                for st in ("sort", "density", "avgflow", "voidage_adhesion", "sand_momentum", "water_momentum"):
                    sim.stage(st, dt)
                sim.stage("integrate", dt)

        outs.append(scenario(sim, sc.n, substep))
        assert sim.check_error() == 0
    for k, v in outs[0][0].items():
        assert np.array_equal(v, outs[1][0][k]), k
    assert np.array_equal(outs[0][1], outs[1][1])
