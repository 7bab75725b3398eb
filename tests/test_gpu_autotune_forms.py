"""sf_autotune times the passes as substeps run them: every kernel form of the neighbour passes that a tuned handle
launches is one that the tuner launched (names as the profiler records them)."""

import re

import pytest

from sph_seepage_flows_gb300 import scenes

pytestmark = pytest.mark.gpu


def _forms(fn):
    """Names (with template arguments) of the neighbour passes that fn launches, with their counts."""
    import torch
    torch.cuda.init()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    out = {}
    for e in prof.key_averages():
        m = re.search(r"(kDensity\w*|kAvgFlow|kVoidageAdhesion|kSandMomentum|kWaterMomentum)(<[^>]*>)?", e.key)
        if m:
            out[m.group(0)] = out.get(m.group(0), 0) + e.count
    return out


@pytest.mark.parametrize("make", [scenes.tiny, lambda: scenes.column_scene("tune", 30_000, 30_000, 3)])
def test_the_tuner_times_the_forms_that_substeps_run(cuda_lib, make):
    pytest.importorskip("torch")
    from sph_seepage_flows_gb300.capi import Simulation
    sim = Simulation(make())
    sim.substeps_fixed(1e-5, 2)
    sim.synchronize()

    def tune():
        sim.autotune(1e-5)
        sim.synchronize()

    def run():
        sim.substeps_fixed(1e-5, 4)
        sim.synchronize()

    _forms(run)  # the profiler's first session may start too late to see anything
    tuned, used = _forms(tune), _forms(run)
    if not used:
        pytest.skip("the profiler records no kernels here")
    assert len(used) == 5 and all(c == 4 for c in used.values()), used
    for name in used:
        assert tuned.get(name, 0) >= 18, (name, tuned)  # three block sizes of six launches each
