"""Which batches step through the buckets: the rule by beads and packing
fraction, and steps and forces on either side of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SORTED = {"ccp": "pair_kernel 2\n", "baseline": "pair_kernel 4\n"}


def _batch(preset, sizes, phi, kernel="", walk=True, chains=None):
    from tfm_gb300.ccpgpu import Batch

    radii = [0.5 * (n / phi) ** (1.0 / 3.0) for n in sizes]
    text = "force_field %s\ncontact_bins 16\n" % preset
    if preset == "ccp":
        text += "number_of_particles %d\nnucleus_radius %.6f\n" % (sizes[0], radii[0])
    b = Batch(text + kernel, sizes, n_chains=chains, radii=radii,
              seeds=list(range(3, 3 + len(sizes))))
    if walk:
        b.generate_initial_condition()
    return b


def _kernels_per_step(b):
    k0 = b.kernel_count()
    b.advance(126)
    k = (b.kernel_count() - k0) // 126
    b.synchronize()
    return k


# beads x (1 + slope x packing fraction) below 44000 (baseline, slope 4) or
# 78000 (ccp, slope 5.3); the walks beyond have more than a quarter of their beads
# in cells of more than 8 (baseline) or 4 (ccp)
@pytest.mark.parametrize("preset,sizes,phi,kernels", [
    ("baseline", [24000], 0.2, 2), ("baseline", [25000], 0.2, 12), ("baseline", [45000], 0.2, 12),
    ("baseline", [40000], 0.02, 2), ("baseline", [42000], 0.02, 12), ("baseline", [24000], 0.3, 12),
    ("baseline", [100] * 240, 0.2, 2), ("baseline", [4000] * 7, 0.2, 12),
    ("ccp", [46000], 0.13, 2), ("ccp", [47000], 0.13, 12), ("ccp", [90000], 0.08, 12),
    ("ccp", [67000], 0.03, 2), ("ccp", [4000] * 11, 0.13, 2), ("ccp", [4000] * 12, 0.13, 12)])
def test_rule(engine_lib, preset, sizes, phi, kernels):
    b = _batch(preset, sizes, phi)
    assert _kernels_per_step(b) == kernels
    b.close()


def _ball(n, a, R):
    """n points of a cubic lattice of side a, those nearest the centre, row by
    row, inside radius R."""
    m = int(np.ceil(R / a))
    k = (np.arange(-m, m + 1) + 0.25) * a
    z, y, x = np.meshgrid(k, k, k, indexing="ij")
    p = np.stack([x.ravel(), y.ravel(), z.ravel()], 1)
    d = (p * p).sum(1)
    p = p[np.sort(np.argsort(d, kind="stable")[:n])]
    assert np.sqrt((p * p).sum(1).max()) < R
    return p.astype(np.float32)


# evenly spread beads beyond the line: 1.5 to 1.9 of ccp's in a cell of 2, 4 of
# the baseline's in one of 2.5; a batch (of chains of one bead: no bonds to strain)
# follows what it is given
@pytest.mark.parametrize("preset,n,phi,a,even", [("ccp", 57000, 0.12, 1.5, 2), ("ccp", 99000, 0.08, 1.7, 2),
                                                 ("baseline", 36000, 0.2, 1.25, 2),
                                                 ("baseline", 42000, 0.2, 1.25, 12)])
def test_path_follows_the_state(engine_lib, preset, n, phi, a, even):
    w = _batch(preset, [n], phi)
    walk = w.positions()
    b = _batch(preset, [n], phi, walk=False, chains=[n])
    c = _batch(preset, [n], phi, SORTED[preset], walk=False, chains=[n])
    for h in (b, c):
        h.set_types(w.types())
        h.set_lbs(w.lbs())
    R = b.system_info(0).nucleus_radius
    ball = _ball(n, a, R - 0.3)
    for x, kernels in ((walk, 12), (ball, even), (walk, 12), (ball, even)):
        b.set_positions(x)
        c.set_positions(x)
        fa, fb = b.forces(), c.forces()
        scale = np.maximum(np.linalg.norm(fb, axis=1), 200.0)
        assert (np.linalg.norm(fa - fb, axis=1) / scale).max() <= 2e-5
        assert _kernels_per_step(b) == kernels
        b.observe()  # the sort of an observation leaves the choice alone
        assert _kernels_per_step(b) == kernels
    assert not b.error_flags()[0][[0, 2]].any()
    assert _kernels_per_step(c) == 12


# on both sides of the line, and the largest batches that step through buckets
@pytest.mark.parametrize("preset,n,phi", [("baseline", 24000, 0.2), ("baseline", 25000, 0.2),
                                          ("ccp", 67000, 0.03), ("ccp", 47000, 0.13)])
def test_steps_and_forces_as_the_sorted_path(engine_lib, preset, n, phi):
    a = _batch(preset, [n], phi)
    b = _batch(preset, [n], phi, SORTED[preset], walk=False)
    b.set_types(a.types())
    b.set_lbs(a.lbs())
    b.set_positions(a.positions())
    for _ in range(2):  # forces from buckets that the steps in between made stale
        fa, fb = a.forces(), b.forces()
        # two FP32 sums over the same terms, each within 1e-5 of max(|F|, 0.1 sum of
        # the terms, 1 kT/sigma); relaxed starts keep the terms of a bead below 2e3
        scale = np.maximum(np.linalg.norm(fb, axis=1), 200.0)
        assert (np.linalg.norm(fa - fb, axis=1) / scale).max() <= 2e-5
        a.run_steps(1)
        b.run_steps(1)
        # |F| dt rounding (forces below 1e3 kT/sigma, relative error < 1e-5) and
        # roundings of a coordinate below 64 sigma
        tol = 1e3 * 1e-5 * a.info().dt + 2.0 ** -24 * 64 * 2
        assert np.abs(a.positions() - b.positions()).max() <= tol
        b.set_positions(a.positions())
    assert not a.error_flags()[0].any()
