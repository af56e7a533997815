"""A refused forces call leaves the caller's array alone."""
import ctypes as C

import numpy as np
import pytest

from helpers import ccp_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["", "pair_kernel 2\n"])
def test_refused_forces_leave_the_array(engine_lib, kernel):
    from tfm_gb300.ccpgpu import ChrSim

    n = 600
    sim = ChrSim(ccp_params(n)[0] + kernel, seed=3)
    sim.generate_initial_condition()
    x = sim.positions()
    k = np.arange(256)
    bad = x.copy()
    bad[:256] = sim.system_info(0).cell_side * (
        0.05 + 0.9 / 7 * np.stack([k % 7, k // 7 % 7, k // 49], 1))  # inside one cell
    sim.set_positions(bad)
    f = np.full((n, 3), 7.0, np.float32)

    def forces():
        return engine_lib.ccpgpu_compute_forces(sim._h, f.ctypes.data_as(C.c_void_p), f.size)

    assert forces() != 0
    assert (f == 7.0).all()
    sim.set_positions(x)
    sim.error_flags(clear=True)
    assert forces() == 0
    assert (f != 7.0).all() and np.isfinite(f).all()
