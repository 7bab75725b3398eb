"""Calls that a caller captures into a graph of its own and replays at any time, which the handle does not see: stages,
fields set and read, the order reset. What the handle knows of its counts and pair copies from call to call may not be
trusted across replays. Compared bit for bit with a handle that runs the same calls directly."""

import ctypes

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu

DT = 1e-4
STAGES = ("sort", "density", "avgflow", "voidage_adhesion", "sand_momentum", "water_momentum", "integrate")
FIELDS = ("id", "key", "pos", "vel", "density", "voidage", "acc")


def stages(sim, names=STAGES):
    for st in names:
        sim.stage(st, DT)


def device_fields(sim, fn, tensors, order):
    from sph_seepage_flows_gb300.capi import FIELDS as TABLE, ORDER
    ids = (ctypes.c_int32 * len(tensors))(*[TABLE[k][0] for k in tensors])
    ptr = (ctypes.c_void_p * len(tensors))(*[t.data_ptr() for t in tensors.values()])
    sim._check(getattr(sim.lib, fn)(sim.h, 0, len(tensors), ids, ORDER[order], ptr, sim.size(0), 1))


class Pair:
    """A handle on a stream that is captured, and one that runs everything directly."""

    def __init__(self, sc):
        import torch
        from sph_seepage_flows_gb300.capi import Simulation
        self.stream = torch.cuda.Stream()
        self.sim, self.ref = Simulation(sc, stream=self.stream.cuda_stream), Simulation(sc)
        self.graph = torch.cuda.CUDAGraph()

    def both(self, fn):
        for s in (self.sim, self.ref):
            fn(s)

    def capture(self, fn):
        import torch
        self.sim.synchronize()
        with torch.cuda.graph(self.graph, stream=self.stream):
            fn(self.sim)

    def replay(self):
        import torch
        with torch.cuda.stream(self.stream):
            self.graph.replay()
        self.sim.synchronize()

    def check(self, names=FIELDS):
        for k in names:
            assert np.array_equal(self.sim.field(k), self.ref.field(k), equal_nan=True), k
        assert np.array_equal(self.sim.cell_table(0), self.ref.cell_table(0))


@pytest.mark.parametrize("side", [None, 6.0])
@pytest.mark.parametrize("before", [("sort",), STAGES, STAGES + ("sort", "density")])
def test_captured_substeps(cuda_lib, before, side):
    """Two substeps in a graph (the buffers are back in place), after any state of the handle; between replays
    positions set, the order reset and substeps run directly. With both forms of the sort."""
    pytest.importorskip("torch")
    sc = scenes.tiny(seed=5) if side is None else scenes.block_scene("wide", (side,) * 3, (6, 7, 5), (7, 5, 6), 0.02, 5)
    p = Pair(sc)
    p.both(lambda s: stages(s, before))

    def two(s):
        stages(s)
        stages(s)

    p.capture(two)
    for turn in range(3):
        p.replay()
        two(p.ref)
        p.check()
        if turn == 0:
            pos = p.ref.field("pos", order="id") + np.float32([0.0, 0.011, 0.0])
            p.both(lambda s: s.set_field("pos", pos, order="id"))
        elif turn == 1:
            p.both(lambda s: s.substeps_fixed(DT, 4))
            p.check()
    p.replay()
    two(p.ref)
    # directly after a replay
    p.both(lambda s: s.step(1.0 / 30.0))
    p.check()
    p.both(lambda s: (s.reset_order(), s.substeps_fixed(DT, 2)))
    p.check()
    assert p.sim.check_error() == 0 and p.ref.check_error() == 0


def test_captured_positions_between_substeps(cuda_lib):
    """A captured write of the positions, replayed between substeps that are run directly."""
    torch = pytest.importorskip("torch")
    p = Pair(scenes.tiny(seed=5))
    p.both(lambda s: s.substeps_fixed(DT, 2))
    n = p.sim.size()
    pos = torch.zeros(n * 3, device="cuda")

    def move(s):
        device_fields(s, "sf_get_fields", {"pos": pos}, "id")
        pos.add_(0.011)
        device_fields(s, "sf_set_fields", {"pos": pos}, "id")

    p.capture(move)
    for _ in range(2):
        p.replay()
        q = p.ref.field("pos", order="id") + np.float32(0.011)
        p.ref.set_field("pos", q, order="id")
        p.both(lambda s: s.substeps_fixed(DT, 2))
        p.check()
        p.both(lambda s: s.adjoint(DT, 2, q, checkpoint_every=2))
        p.check(("id", "pos", "vel"))


def test_captured_integration_between_stages(cuda_lib):
    """A captured integration, replayed between a sort and a density pass that are run directly; and one captured alone
    whose next sort is run directly."""
    pytest.importorskip("torch")
    p = Pair(scenes.tiny(seed=5))
    p.both(stages)
    p.both(lambda s: stages(s, STAGES[:6]))
    p.capture(lambda s: s.stage("integrate", DT))
    for _ in range(2):
        p.replay()
        p.ref.stage("integrate", DT)
        p.both(lambda s: stages(s, STAGES[1:6]))
        p.check(("id", "pos", "vel", "density", "acc"))
        p.replay()
        p.ref.stage("integrate", DT)
        p.both(lambda s: (stages(s), stages(s, STAGES[:6])))
        p.check()
