"""Per-kernel times name the kernels that the batch steps with."""
import numpy as np
import pytest

from helpers import baseline_params, ccp_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset,kernel", [("ccp", ""), ("ccp", "pair_kernel 2\n"), ("baseline", ""),
                                           ("baseline", "pair_kernel 4\n")])
def test_times_of_the_kernels_that_step(engine_lib, preset, kernel):
    from tfm_gb300.ccpgpu import ChrSim

    n = 1500
    text = (ccp_params(n)[0] if preset == "ccp" else baseline_params(n)) + kernel
    a, b = ChrSim(text, seed=4), ChrSim(text, seed=4)
    a.generate_initial_condition()
    b.load_checkpoint_bytes(a.checkpoint())
    b.set_lbs(a.lbs())
    assert np.array_equal(a.positions(), b.positions()) and a.info().step == b.info().step
    for h in (a, b):
        h.reset_observables()
    step, k0 = a.info().step, a.kernel_count()
    reps = 4  # the count arrays of the buckets end in another phase
    t = a.kernel_times(reps=reps)
    kernels = a.kernel_count() - k0
    assert list(t) == list(a.KERNELS)
    assert (t["pair"] == 0.0) == (kernel == "")
    assert all(v > 0.0 for k, v in t.items() if k != "pair" or kernel)
    # two stage kernels a step and an observation (count, scan, scatter, contacts,
    # observe) each time, against twelve and two
    assert kernels <= reps * (9 if kernel == "" else 14) + 3
    assert a.info().step == step + reps and a.info().frames_observed == reps
    # the state is the one that plain steps reach
    b.run_steps(reps)
    assert np.abs(a.positions() - b.positions()).max() <= 1e-4
    a.run_steps(3)
    assert not a.error_flags()[0].any()
