"""The autotuner's choice of the bucket path."""
import pytest

from helpers import baseline_params, ccp_params

pytestmark = pytest.mark.gpu


def _sim(preset, n):
    from tfm_gb300.ccpgpu import ChrSim

    sim = ChrSim(ccp_params(n)[0] if preset == "ccp" else baseline_params(n), seed=4)
    sim.generate_initial_condition()
    return sim


def _kernels_per_step(sim):
    k0 = sim.kernel_count()
    sim.advance(126)
    k = (sim.kernel_count() - k0) // 126
    sim.synchronize()
    return k


# Steps of the bucket path take a quarter of the sorted path's time at 1024
# beads; a number of steps that is no multiple of three starts every run in
# another phase of the count arrays, with a graph of its own.
@pytest.mark.parametrize("reps", [1, 2, 3, 5])
@pytest.mark.parametrize("preset", ["ccp", "baseline"])
def test_any_number_of_steps_finds_the_buckets(engine_lib, preset, reps):
    sim = _sim(preset, 1024)
    assert sim.autotune(reps=reps)["buckets"] == 1
    assert _kernels_per_step(sim) == 2
