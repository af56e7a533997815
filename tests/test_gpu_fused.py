"""The one-kernel Heun stages of small batches (tfm_gb300/csrc/fused.cuh)
against the FP64 oracle and the sorted path, at the sizes where a rule or a
tile ends."""
import numpy as np
import pytest

from helpers import baseline_params, ccp_params, heads_of

pytestmark = pytest.mark.gpu

# a text that names the pair kernel keeps the sorted path
SORTED = {"ccp": "pair_kernel 2\n", "baseline": "pair_kernel 4\n"}


def _text(preset, n):
    return ccp_params(n)[0] if preset == "ccp" else baseline_params(n)


def _pair(text, preset, seed):
    from tfm_gb300.ccpgpu import ChrSim

    a = ChrSim(text, seed=seed)
    b = ChrSim(text + SORTED[preset], seed=seed)
    a.generate_initial_condition()
    return a, b


def _same_start(a, b):
    b.set_types(a.types())
    b.set_lbs(a.lbs())
    b.set_positions(a.positions())


# 32, 16, 8 and 4 lanes a bead (3648 and 7296 beads end the first two on 152
# SMs), full and partial last tiles of each, and the largest batch of the path
@pytest.mark.parametrize("preset,n", [("ccp", 65), ("ccp", 3647), ("ccp", 3649), ("ccp", 7297),
                                      ("ccp", 49153), ("baseline", 577), ("baseline", 3648),
                                      ("baseline", 7296), ("baseline", 7297), ("baseline", 45000)])
def test_fused_steps_as_the_sorted_path(engine_lib, preset, n):
    a, b = _pair(_text(preset, n), preset, 5)
    _same_start(a, b)
    a.run_steps(1)
    b.run_steps(1)
    # one step differs by the order of the pair sums only: |F| dt rounding,
    # forces of a relaxed start below 1e3 kT/sigma with relative error < 1e-5
    # and one rounding of a coordinate below 64 sigma
    tol = 1e3 * 1e-5 * a.info().dt + 2.0 ** -24 * 64 * 2
    assert np.abs(a.positions() - b.positions()).max() <= tol
    a.run_steps(4)
    b.run_steps(4)
    assert np.abs(a.positions() - b.positions()).max() <= 20 * tol
    assert not a.error_flags()[0].any()


@pytest.mark.parametrize("preset", ["ccp", "baseline"])
def test_fused_steps_against_the_oracle(engine_lib, orc, preset):
    from tfm_gb300.ccpgpu import ChrSim

    n = 777
    sim = ChrSim(_text(preset, n) + "number_of_chains 3\n", seed=8)
    sim.generate_initial_condition()
    x = sim.positions()
    ff = orc.ccp_ff() if preset == "ccp" else orc.baseline_ff()
    fl = orc.flags_from_types(sim.types(), heads_of(sim), preset)
    ref = orc.run(x, fl, sim.lbs(), ff, orc.geo_vec(sim.system_info(0).nucleus_radius, csl=2.5), 8, 0, 10)
    sim.run_steps(10)
    # 20 roundings of coordinates below 16 sigma, and FP32 forces
    assert np.abs(sim.positions() - ref).max() <= 20 * 2.0 ** -24 * 16 + 20 * 1e-2 * sim.info().dt


def test_fused_batch_with_observation(engine_lib):
    """Systems of different size side by side, an observed step between."""
    from tfm_gb300.ccpgpu import Batch

    sizes, text = [1, 2, 31, 700, 1025], "force_field baseline\ncontact_bins 16\n"
    radii = [4.0, 4.0, 5.0, 8.0, 9.0]
    a = Batch(text, sizes, radii=radii, seeds=[3, 4, 5, 6, 7])
    b = Batch(text + SORTED["baseline"], sizes, radii=radii, seeds=[3, 4, 5, 6, 7])
    a.generate_initial_condition()
    _same_start(a, b)
    for h in (a, b):
        h.reset_observables()
        h.run_steps(7, observe_every=5)
    assert np.abs(a.positions() - b.positions()).max() <= 1e-4
    assert a.info().frames_observed == b.info().frames_observed == 2
    for s in range(len(sizes)):
        d = np.abs(a.contact_counts(s) - b.contact_counts(s)).sum()
        assert d <= 2  # a pair at the cutoff after five steps may fall on either side
    # forces and another run after the observation start from the same state
    fa, fb = a.forces(), b.forces()
    assert np.abs(fa - fb).max() <= 1e-3 * max(1.0, np.abs(fb).max())
    a.run_steps(2)
    b.run_steps(2)
    assert np.abs(a.positions() - b.positions()).max() <= 2e-4


def test_fused_overfull_cells(engine_lib):
    """More beads in a cell than it has slots: the overflow list takes them."""
    from tfm_gb300.ccpgpu import ChrSim

    n = 600
    a, b = _pair(baseline_params(n), "baseline", 2)
    k = np.arange(64)
    x = a.positions()
    # 64 beads 0.62 sigma apart inside the cell [0, 2.5)^3, and as many around
    # the corner of eight cells
    cube = 0.62 * np.stack([k % 4, k // 4 % 4, k // 16], 1)
    cube = cube + 0.03 * np.random.default_rng(1).standard_normal((64, 3))
    x[:64] = cube + 0.2
    x[64:128] = cube - [0.93, 0.93, 3.43]
    a.set_positions(x)
    _same_start(a, b)
    a.run_steps(1)
    b.run_steps(1)
    # Up to 26 pair terms of 3e4 kT/sigma and 1e-6 relative error, against
    # sums that the jitter leaves at 1e3 or more: the capped displacement of
    # 0.1 sigma turns by less than 1e-3 in either stage, a hundred times that
    # for a bead whose sum is 1 % of it
    d = np.abs(a.positions() - b.positions()).max(1)
    assert np.median(d) <= 1e-4 and d.max() <= 2e-2
    assert not a.error_flags()[0][[0, 2]].any()


@pytest.mark.parametrize("preset,n", [("ccp", 65), ("ccp", 3649), ("ccp", 49153), ("baseline", 7297),
                                      ("baseline", 45000)])
def test_fused_forces_as_the_sorted_path(engine_lib, preset, n):
    a, b = _pair(_text(preset, n), preset, 5)
    _same_start(a, b)
    fa, fb = a.forces(), b.forces()
    # two FP32 sums over the same terms, each within 1e-5 of max(|F|, 0.1 sum of
    # the terms, 1 kT/sigma); relaxed starts keep the terms of a bead below 2e3
    scale = np.maximum(np.linalg.norm(fb, axis=1), 200.0)
    assert (np.linalg.norm(fa - fb, axis=1) / scale).max() <= 2e-5


def _status(call):
    from tfm_gb300.ccpgpu import CcpError

    try:
        call()
    except CcpError as e:
        return e.code, str(e)
    return 0, ""


# The sort's cells count up to 255 beads (of a class, in the baseline field's
# two grids); more are refused, by either path.
@pytest.mark.parametrize("preset,m,mixed,refused", [("ccp", 255, False, False), ("ccp", 256, False, True),
                                                    ("ccp", 256, True, True), ("baseline", 255, False, False),
                                                    ("baseline", 256, False, True),
                                                    ("baseline", 288, True, False)])
def test_fused_refuses_what_the_sort_refuses(engine_lib, preset, m, mixed, refused):
    from tfm_gb300.ccpgpu import ChrSim

    n = 600
    a = ChrSim(_text(preset, n), seed=3)
    b = ChrSim(_text(preset, n) + SORTED[preset], seed=3)
    side = a.system_info(0).cell_side
    k = np.arange(m)
    x = np.zeros((n, 3), np.float32)
    x[:m] = side * (0.05 + 0.9 / 7 * np.stack([k % 7, k // 7 % 7, k // 49], 1))  # inside one cell
    k = np.arange(n - m)
    x[m:] = -0.3 - 0.55 * np.stack([k % 7, k // 7 % 7, k // 49], 1)
    types = np.arange(n, dtype=np.int32) % 2 if mixed else np.ones(n, np.int32)
    for h in (a, b):
        h.set_types(types)
        h.set_lbs(a.lbs())
        h.set_positions(x)
        code, message = _status(h.forces)
        assert (code != 0) == refused and ("cell list" in message) == refused
        h.error_flags(clear=True)
        if refused:
            assert _status(lambda: h.run_steps(1))[0] == code


@pytest.mark.parametrize("preset", ["ccp", "baseline"])
def test_fused_escape_flag_as_the_sorted_path(engine_lib, preset):
    a, b = _pair(_text(preset, 700), preset, 4)
    _same_start(a, b)
    s = b.system_info(0)
    edge = s.cells_per_side / 2 * s.cell_side
    x = a.positions()
    for dx, escaped in ((-0.01, 0), (0.01, 1)):
        x[5] = [edge + dx, 0.3, 0.2]
        for h in (a, b):
            h.set_positions(x)
            _status(h.forces)
            assert h.error_flags(clear=True)[0][1] == escaped
