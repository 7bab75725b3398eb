"""The adjoint pair kernels take 8, 4, 2 or 1 threads per particle by the
number of slots. Around the sizes where that changes, the gradients of the
automatic choice are those of one thread per particle up to the order of the
sums.

Tolerance: a particle adds up to a few hundred FP32 terms (96 listed
neighbours of each kind, several levels), in another order by the lane, so a
sum moves by about sqrt(300) * 2^-24 = 1e-6 of its terms' size; the terms
cancel by up to one digit or two: 1e-4 in the 2-norm."""

import numpy as np
import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu

DT = 2e-4
TOL = 1e-4


@pytest.mark.parametrize("per_sm", [512, 1024, 2048, 4096])
@pytest.mark.parametrize("above", [False, True], ids=["below", "above"])
def test_gradients_do_not_depend_on_the_lanes(cuda_lib, per_sm, above):
    import torch
    from sph_seepage_flows_gb300.capi import Simulation
    slots = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    n = int(slots * (1.07 if above else 0.93))   # the scene's counts come out within a layer of these
    sc = scenes.embankment_scene("lanes", n // 3, n - n // 3, seed=4)
    target = sc.pos + np.random.default_rng(2).uniform(-1e-3, 1e-3, sc.pos.shape).astype(np.float32)
    got = []
    for lanes in (0, 1):
        sim = Simulation(sc)
        sim.set_lanes(lanes)
        got.append(sim.adjoint(DT, 1, target))
        sim.close()
    auto, one = got
    for key in ("grad_pos0", "grad_vel0", "grad_params"):
        a, b = auto[key].astype(np.float64), one[key].astype(np.float64)
        assert np.isfinite(b).all()
        assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b), key
    assert abs(float(auto["loss"][0]) - float(one["loss"][0])) <= TOL * abs(float(one["loss"][0]))
