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


@pytest.mark.parametrize("preset,kernel,per_step", [("ccp", "", 2), ("baseline", "", 2),
                                                    ("ccp", "pair_kernel 2\n", 12),
                                                    ("baseline", "pair_kernel 4\n", 12)])
def test_a_failed_search_changes_nothing(engine_lib, preset, kernel, per_step):
    """An error flag that is already set makes the search fail at its first
    candidate (the positions themselves are in order)."""
    import numpy as np

    from tfm_gb300.ccpgpu import CcpError, ChrSim

    n = 700
    sim = ChrSim((ccp_params(n)[0] if preset == "ccp" else baseline_params(n)) + kernel, seed=4)
    sim.generate_initial_condition()
    sim.run_steps(10)
    x = sim.positions()
    before = [getattr(sim.system_info(0), k) for k in ("cell_side", "cells_per_side")]
    bad = x.copy()
    k = np.arange(300)  # all inside one cell
    bad[:300] = before[0] * (0.05 + 0.9 / 7 * np.stack([k % 7, k // 7 % 7, k // 49], 1))
    pt = sim.types()
    sim.set_types(pt & ~1)  # of one class
    sim.set_positions(bad)
    sim.set_types(pt)
    sim.set_positions(x)
    step = sim.info().step
    with pytest.raises(CcpError, match="cell list"):
        sim.autotune(reps=3)
    sim.error_flags(clear=True)
    assert [getattr(sim.system_info(0), k) for k in ("cell_side", "cells_per_side")] == before
    assert np.array_equal(sim.positions(), x) and sim.info().step == step
    assert _kernels_per_step(sim) == per_step
    assert sim.autotune(reps=3)["buckets"] == (1 if per_step == 2 else 0)
