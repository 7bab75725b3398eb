"""Particles parked by a mass of 0 keep their ids and, through every sort, their slot order before the blank slots,
in both forms of the sort stage: checked against numpy's stable order, by the reads by id, and by setting the masses
back and running on."""

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes
from test_gpu_cell_sort import keys_of, make_scene

pytestmark = pytest.mark.gpu


def park(n, rng):
    """Ids to park: singles everywhere, a whole warp, a whole block and some of the last warp, as far as n goes."""
    out = np.zeros(n, bool)
    out[rng.permutation(n)[:max(1, n // 20)]] = True
    out[n - 1 - n // 7 % 5] = True
    if n > 600:
        out[64:96] = True
        out[256:512] = True
    return out


@pytest.mark.parametrize("sizes, side, spare", [
    ((5,), 0.4, 0), ((255, 256, 257), 0.4, 0), ((1000,), 0.4, 5000), ((20011,), 1.3, 0), ((900, 3000), 0.4, 40),
    ((1000, 700), 0.4, 400000), ((1500,), 6.0, 300)])
def test_parked_particles_stay_in_slot_order(cuda_lib, sizes, side, spare):
    from sph_seepage_flows_gb300.capi import Simulation
    scs = [make_scene(n, side, 20 + k) for k, n in enumerate(sizes)]
    sim = Simulation(scs, capacity=[sc.n + spare for sc in scs])
    order = [np.arange(sc.n) for sc in scs]
    pos, mass = [sc.pos for sc in scs], [sc.mass for sc in scs]
    rng = np.random.default_rng(2)
    for turn in range(4):
        for s, sc in enumerate(scs):  # others each turn; those of the turn before are set back
            mass[s] = np.where(park(sc.n, rng) & (turn < 3), np.float32(0), sc.mass)
            pos[s] = np.where(rng.random((sc.n, 1)) < 0.2, rng.uniform(0, side, (sc.n, 3)), pos[s]).astype(np.float32)
            sim.set_fields({"mass": mass[s], "pos": pos[s]}, order="id", scene=s)
        for again in range(2):
            sim.stage("sort")
            for s, sc in enumerate(scs):
                keys, cells = keys_of(sc, pos[s])
                keys = np.where(mass[s] == 0, cells, keys)
                order[s] = order[s][np.argsort(keys[order[s]], kind="stable")]
                assert np.array_equal(sim.field("id", scene=s), order[s]), (turn, again, s)
                assert np.array_equal(sim.field("key", scene=s), keys[order[s]]), (turn, again, s)
                assert np.array_equal(sim.field("pos", order="id", scene=s), pos[s]), (turn, again, s)
                assert np.array_equal(sim.field("mass", order="id", scene=s), mass[s]), (turn, again, s)
                table = np.searchsorted(keys[order[s]], np.arange(cells + 1))
                assert np.array_equal(sim.cell_table(0, scene=s), table), (turn, again, s)
    assert sim.check_error() == 0


@pytest.mark.parametrize("block", [0, 32])
def test_parked_particles_through_substeps(cuda_lib, block):
    """Counts left by the integrator (also in small blocks), particles added while others are parked, masses set back:
    parked particles keep their state and the run goes on, the same on every handle."""
    from sph_seepage_flows_gb300.capi import Simulation
    outs = []
    for _ in range(3):
        sc = scenes.tiny(seed=6)
        sim = Simulation(sc, capacity=sc.n + 30)
        sim.set_tuning(block)
        rng = np.random.default_rng(4)
        off = park(sc.n, rng)
        sim.substeps_fixed(1e-4, 3)
        state = {k: sim.field(k, order="id") for k in ("pos", "mass", "label")}
        sim.set_field("mass", np.where(off, np.float32(0), state["mass"]), order="id")
        sim.substeps_fixed(1e-4, 3)
        sim.add_sph_particles(rng.uniform(0.1, 0.3, (20, 3)), [0, 0, 1], [0, 0, 0], float(sc.params.sph_mass), 0.01)
        sim.substeps_fixed(1e-4, 3)
        sim.step(1.0 / 30.0)
        ids, mass = sim.field("id"), sim.field("mass", order="id")
        assert np.array_equal(np.sort(ids), np.arange(sc.n + 20))
        assert np.array_equal(mass[:sc.n] == 0, off) and not (mass[sc.n:] == 0).any()
        pos = sim.field("pos", order="id")
        assert np.array_equal(pos[:sc.n][off], state["pos"][off])
        sim.set_field("mass", np.concatenate([state["mass"], mass[sc.n:]]), order="id")
        sim.set_field("label", np.concatenate([state["label"], np.zeros(20, np.int32)]), order="id")
        sim.substeps_fixed(1e-4, 3)
        outs.append({k: sim.field(k) for k in ("id", "pos", "vel", "density", "mass")})
        assert np.array_equal(np.sort(outs[-1]["id"]), np.arange(sc.n + 20))
        assert not (outs[-1]["mass"] == 0).any()
        assert sim.check_error() == 0
    for o in outs[1:]:
        for k, v in o.items():
            assert np.array_equal(v, outs[0][k]), k


@pytest.mark.parametrize("side", [0.4, 6.0])
def test_particles_parked_between_stages_by_hand(cuda_lib, side):
    """Masses set, taken back and particles added right before an integration run by hand: the sort after it is numpy's
    stable order of what the integration left, in both forms."""
    from sph_seepage_flows_gb300.capi import Simulation
    sc = make_scene(2000, side, 7)
    sim = Simulation(sc, capacity=sc.n + 200)
    rng = np.random.default_rng(3)
    for turn in range(5):
        sim.stage("sort")
        n = sim.size()
        if turn:
            mass = sim.field("mass", order="id")
            mass[:sc.n] = np.where(park(sc.n, rng) & (turn < 4), np.float32(0), sc.mass)
            sim.set_field("mass", mass, order="id")
        if turn in (0, 2):
            sim.add_sph_particles(rng.uniform(0.05, 0.35, (30, 3)), [0, 0, 1], [0, 0, 0], float(sc.params.sph_mass), 0.01)
        ids = sim.field("id")
        assert np.array_equal(np.sort(ids), np.arange(sim.size())) and sim.size() - n == 30 * (turn in (0, 2))
        sim.stage("integrate", 1e-6)
        mass = sim.field("mass", order="id")
        sim.stage("sort")
        keys, cells = keys_of(sc, sim.field("pos", order="id"))
        keys = np.where(mass == 0, cells, keys)
        want = ids[np.argsort(keys[ids], kind="stable")]
        assert np.array_equal(sim.field("id"), want), turn
        assert np.array_equal(sim.field("key"), keys[want]), turn
        assert np.array_equal(sim.cell_table(0), np.searchsorted(keys[want], np.arange(cells + 1))), turn
