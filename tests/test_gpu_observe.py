"""Observation kernels at the sizes where their tiles and lane rules end: the
distance sums of all chains in one launch, and the contact pass."""
import numpy as np
import pytest

from helpers import ccp_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chains", [(3, 3), (64, 1), (257, 1), (600, 7), (1026, 2), (2051, 3)])
def test_distance_sums_of_every_chain(engine_lib, orc, n, chains):
    """Chains of one to a few hundred beads: below, at and above a CTA's 128
    separations and 256 first beads."""
    from tfm_gb300.ccpgpu import ChrSim

    txt = ccp_params(n, cvf=0.05)[0] + "number_of_chains %d\n" % chains
    sim = ChrSim(txt, seed=3)
    sim.generate_initial_condition()
    x = sim.positions()
    sim.reset_observables()
    sim.observe(with_sdist=True)
    sim.observe(with_sdist=True)
    L = n // chains
    for c in range(chains):
        first = c * L
        last = n if c == chains - 1 else first + L
        _, d = sim.separation_counts(c, last - first)
        # FP32 sums over at most 256 distances below 100, twice
        ref = 2 * orc.sdist(x[first:last])
        assert np.abs(d - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max())


# eight lanes a bead below 16384 beads, four below 65536, two below 262144
@pytest.mark.parametrize("preset,n", [("ccp", 70), ("baseline", 1500), ("ccp", 16385),
                                      ("baseline", 16384), ("baseline", 65537)])
def test_contact_counts_by_lanes(engine_lib, preset, n):
    """Counts of the default layout against another one: cells of the whole
    cutoff and one grid (ccp) or the full-stencil sort's kernel (baseline)."""
    from tfm_gb300.ccpgpu import ChrSim

    if preset == "ccp":
        txt, other = ccp_params(n)[0], "cell_side 2.5\n"
    else:
        txt, other = "force_field baseline\nnumber_of_particles %d\ncontact_bins 64\n" % n, "pair_kernel 0\n"
    a, b = ChrSim(txt, seed=4), ChrSim(txt + other, seed=4)
    a.generate_initial_condition()
    b.set_types(a.types())
    b.set_lbs(a.lbs())
    b.set_positions(a.positions())
    for h in (a, b):
        h.reset_observables()
        h.observe()
    assert np.array_equal(a.contact_counts(0), b.contact_counts(0))
    assert np.array_equal(a.separation_counts(0, n)[0], b.separation_counts(0, n)[0])
    assert a.contact_counts(0).sum() > 0
    assert np.array_equal(a.overlaps(), b.overlaps())
