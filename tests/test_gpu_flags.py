"""Device error flags that a caller has cleared come back with every call that
looks at the positions, on the bucket path and on the sorted one."""
import numpy as np
import pytest

from helpers import baseline_params, ccp_params

pytestmark = pytest.mark.gpu

CALLS = {"forces": lambda h: h.forces(), "observe": lambda h: h.observe(),
         "analysis_frame": lambda h: h.analysis_frame(), "overlaps": lambda h: h.overlaps()}


def _sim(preset, kernel, n=700):
    from tfm_gb300.ccpgpu import ChrSim

    sim = ChrSim((ccp_params(n)[0] if preset == "ccp" else baseline_params(n)) + kernel, seed=4)
    sim.generate_initial_condition()
    return sim


PATHS = [("ccp", ""), ("ccp", "pair_kernel 2\n"), ("baseline", ""), ("baseline", "pair_kernel 4\n")]


@pytest.mark.parametrize("call", list(CALLS))
@pytest.mark.parametrize("preset,kernel", PATHS)
def test_escape_is_flagged_by_every_call(engine_lib, preset, kernel, call):
    sim = _sim(preset, kernel)
    s = sim.system_info(0)
    x = sim.positions()
    x[5] = [s.cells_per_side / 2 * s.cell_side + 0.01, 0.3, 0.2]
    sim.set_positions(x)
    assert sim.error_flags(clear=True)[0][1] == 1
    for _ in range(3):
        CALLS[call](sim)
        assert sim.error_flags(clear=True)[0][1] == 1
    x[5] = 0.1
    sim.set_positions(x)
    CALLS[call](sim)
    assert sim.error_flags()[0][1] == 0


@pytest.mark.parametrize("call", list(CALLS))
@pytest.mark.parametrize("preset,kernel", PATHS)
def test_overfull_cell_is_refused_by_every_call(engine_lib, preset, kernel, call):
    from tfm_gb300.ccpgpu import CcpError

    sim = _sim(preset, kernel)
    x = sim.positions()
    side = sim.system_info(0).cell_side
    k = np.arange(256)
    x[:256] = side * (0.05 + 0.9 / 7 * np.stack([k % 7, k // 7 % 7, k // 49], 1))  # inside one cell
    pt = sim.types()
    pt[:256] &= ~1  # of one class
    sim.set_types(pt)
    sim.set_positions(x)
    sim.error_flags(clear=True)
    for _ in range(3):
        with pytest.raises(CcpError):
            CALLS[call](sim)
        assert sim.error_flags(clear=True)[0][2] == 1
