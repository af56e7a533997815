"""Trajectories of the sorted path against the FP64 oracle. A text that names
the pair kernel steps through it at sizes that the oracle can follow; larger
batches do so by default."""
import numpy as np
import pytest

from helpers import baseline_params, ccp_params

pytestmark = pytest.mark.gpu

KERNEL = {"ccp": "pair_kernel 2\n", "baseline": "pair_kernel 4\n"}


def _kernels_per_step(sim, steps):
    """Kernels of a captured step: 12 on the sorted path, 2 on the bucket path."""
    k0 = sim.kernel_count()
    sim.run_steps(steps)
    return (sim.kernel_count() - k0) // steps


@pytest.mark.parametrize("path,kernels", [("sorted", 12), ("buckets", 2)])
@pytest.mark.parametrize("preset", ["ccp", "baseline"])
def test_1000_steps_match_the_oracle(engine_lib, orc, preset, path, kernels):
    """Same start and noise: max |dr| < 2e-3 sigma after 1000 Heun steps, FP32
    rounding amplified by the chaotic dynamics (the bound of the other paths)."""
    from tfm_gb300.ccpgpu import ChrSim

    text = ccp_params(1024, laf=0.3)[0] if preset == "ccp" else baseline_params(1024)
    sim = ChrSim(text + (KERNEL[preset] if path == "sorted" else ""), seed=1234)
    sim.generate_initial_condition()
    x0, pt, lbs, step0 = sim.positions(), sim.types(), sim.lbs(), sim.info().step
    assert _kernels_per_step(sim, 1000) == kernels
    ff = orc.ccp_ff() if preset == "ccp" else orc.baseline_ff()
    geo = orc.geo_vec(sim.system_info(0).nucleus_radius, csl=2.0 if preset == "ccp" else 2.5)
    ref = orc.run(x0, orc.flags_from_types(pt, [0], preset), lbs, ff, geo, 1234, step0, 1000, prec=64)
    assert np.linalg.norm(sim.positions() - ref, axis=1).max() < 2e-3


@pytest.mark.parametrize("preset", ["ccp", "baseline"])
def test_batch_matches_single_systems(engine_lib, preset):
    """200 sorted steps of a batch and of its systems alone (other tiles and
    lanes), as the bucket path's test bounds them."""
    from tfm_gb300.ccpgpu import Batch

    sizes, seeds = [1024, 1536, 2048], [5, 6, 7]
    text = "force_field %s\ncontact_bins 64\n" % preset + KERNEL[preset]
    radii = [0.5 * (n / 0.1) ** (1.0 / 3.0) for n in sizes]
    if preset == "ccp":
        text += "number_of_particles %d\nnucleus_radius %.6f\n" % (sizes[0], radii[0])
    b = Batch(text, sizes, radii=radii, seeds=seeds)
    b.generate_initial_condition()
    x0, pt, step0 = b.positions(), b.types(), b.info().step
    assert _kernels_per_step(b, 200) == 12
    xb, off = b.positions(), 0
    for k, n in enumerate(sizes):
        s = Batch(text, [n], radii=[radii[k]], seeds=[seeds[k]])
        s.generate_initial_condition()
        assert s.info().step == step0 and np.array_equal(s.types(), pt[off:off + n])
        s.set_positions(x0[off:off + n])
        s.run_steps(200)
        assert np.abs(s.positions() - xb[off:off + n]).max() < 1e-3
        off += n


def test_default_of_a_large_system_matches_the_oracle(engine_lib, orc):
    """Ten default steps of a system above the bucket path's limit."""
    from tfm_gb300.ccpgpu import ChrSim

    n = 40000
    sim = ChrSim(baseline_params(n, "number_of_chains 8\n"), seed=2)
    sim.generate_initial_condition()
    x0, lbs, step0 = sim.positions(), sim.lbs(), sim.info().step
    fl = orc.flags_from_types(sim.types(), [c * (n // 8) for c in range(8)], "baseline")
    assert _kernels_per_step(sim, 10) == 12
    ref = orc.run(x0, fl, lbs, orc.baseline_ff(), orc.geo_vec(sim.system_info(0).nucleus_radius, csl=2.5),
                  2, step0, 10)
    # 20 roundings of coordinates below 32 sigma, and FP32 forces within 1e-2
    assert np.abs(sim.positions() - ref).max() <= 20 * 2.0 ** -24 * 32 + 20 * 1e-2 * sim.info().dt


def test_forces_of_the_tuned_sorted_path(engine_lib):
    """The tuner's pair kernel, cells, tile and lanes give the same forces."""
    from tfm_gb300.ccpgpu import Batch

    b = Batch("force_field baseline\ncontact_bins 64\npair_kernel 4\n", [1100, 1500, 2600, 5000],
              seeds=[1, 2, 3, 4])
    b.generate_initial_condition()
    b.run_steps(50)
    before = b.forces()
    assert b.autotune(reps=3)["buckets"] == 0
    after = b.forces()
    # two FP32 sums over the same terms, each within 1e-5 of max(|F|, 0.1 sum of
    # the terms, 1 kT/sigma); relaxed starts keep the terms of a bead below 2e3
    scale = np.maximum(np.linalg.norm(before, axis=1), 200.0)
    assert (np.linalg.norm(after - before, axis=1) / scale).max() <= 2e-5
