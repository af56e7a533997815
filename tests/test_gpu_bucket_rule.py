"""Which batches step through the buckets: the rule by beads and packing
fraction, and steps and forces on either side of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SORTED = {"ccp": "pair_kernel 2\n", "baseline": "pair_kernel 4\n"}


def _batch(preset, sizes, phi, kernel="", walk=True):
    from tfm_gb300.ccpgpu import Batch

    radii = [0.5 * (n / phi) ** (1.0 / 3.0) for n in sizes]
    text = "force_field %s\ncontact_bins 16\n" % preset
    if preset == "ccp":
        text += "number_of_particles %d\nnucleus_radius %.6f\n" % (sizes[0], radii[0])
    b = Batch(text + kernel, sizes, radii=radii, seeds=list(range(3, 3 + len(sizes))))
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
# 78000 (ccp, slope 5.3)
@pytest.mark.parametrize("preset,sizes,phi,kernels", [
    ("baseline", [24000], 0.2, 2), ("baseline", [25000], 0.2, 12), ("baseline", [45000], 0.2, 12),
    ("baseline", [40000], 0.02, 2), ("baseline", [42000], 0.02, 12), ("baseline", [24000], 0.3, 12),
    ("baseline", [100] * 240, 0.2, 2), ("baseline", [100] * 250, 0.2, 12),
    ("ccp", [46000], 0.13, 2), ("ccp", [47000], 0.13, 12), ("ccp", [90000], 0.08, 12),
    ("ccp", [67000], 0.03, 2), ("ccp", [4000] * 11, 0.13, 2), ("ccp", [4000] * 12, 0.13, 12)])
def test_rule(engine_lib, preset, sizes, phi, kernels):
    b = _batch(preset, sizes, phi)
    assert _kernels_per_step(b) == kernels
    b.close()


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
