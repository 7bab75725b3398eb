"""State gradients take no device memory of their own: a run that returns them fits where one without them did, and
their values do not depend on what the handle's buffers held before."""

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_state_gradients_take_no_device_memory(cuda_lib):
    torch = pytest.importorskip("torch")
    from sph_seepage_flows_gb300.capi import Simulation
    sc = scenes.column_scene("memory", 100_000, 100_000, 3)
    sim = Simulation(sc)
    target = (sc.pos + np.float32(1e-3)).astype(np.float32)

    def run(checkpoint_every, **kw):
        sim.reset_order()
        sim.set_fields({"pos": sc.pos, "vel": sc.vel, "max_saturation": np.zeros(sc.n, np.float32)}, order="sorted")
        out = sim.adjoint(1e-5, 3, target, checkpoint_every=checkpoint_every, **kw)
        torch.cuda.synchronize()
        return out, torch.cuda.mem_get_info()[0]

    # both buffer sets' graphs, and the staging of the fields, by two runs without state gradients
    for every in (3, 2, 3, 2):
        _, before = run(every, want_state_grads=False)
    outs = []
    for every in (3, 2, 2):
        out, after = run(every, want_state_grads=True)
        assert after == before, (before, after)
        outs.append(out)
    for k in ("grad_pos0", "grad_vel0"):
        assert np.any(outs[0][k] != 0)
        assert np.array_equal(outs[1][k], outs[2][k]), k
