"""The bond force next to its zero: (d^2 - l_0^2) keeps its relative precision
where bonds are within 1e-7 .. 1e-5 of their length l_0."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset,kernel", [("ccp", ""), ("ccp", "pair_kernel 2\n"), ("baseline", ""),
                                           ("baseline", "pair_kernel 4\n")])
def test_bond_force_near_its_zero(engine_lib, orc, preset, kernel):
    from tfm_gb300.ccpgpu import ChrSim

    ff = orc.ccp_ff() if preset == "ccp" else orc.baseline_ff()
    sim = ChrSim("force_field %s\nnumber_of_particles 2\nnucleus_radius 20\nnumber_of_lbs 0\n" % preset
                 + kernel, seed=1)
    rng = np.random.default_rng(5)
    seen = 0
    while seen < 150:
        u = rng.standard_normal(3)
        u /= np.linalg.norm(u)
        x = rng.uniform(-2.0, 2.0, (2, 3))
        x[1] = x[0] + u * (1.0 + rng.choice([-1, 1]) * 10.0 ** rng.uniform(-7, -5))
        x = x.astype(np.float32)
        v = x[1].astype(np.float64) - x[0]
        d2, l0 = v @ v, ff["l_0"]
        s = d2 - l0 * l0
        if not 1e-7 <= abs(s) <= 1e-5:
            continue
        seen += 1
        sim.set_positions(x)
        f = sim.forces()
        d = np.sqrt(d2)
        ref = ff["k_e"] * s / ((d + l0) * d) * v
        # The two beads feel their bond only. s is formed by error-free
        # products and sums whose errors, below 1.3e-7 in all, are added with
        # seven roundings (2^-24 each): 6e-14; then one rounding of s, and ten
        # of the factors (the reciprocal root has two ulps)
        tol = ff["k_e"] / (2.0 * l0) * 1e-13 + 11 * 2.0 ** -23 * np.linalg.norm(ref)
        assert np.abs(f[1] + ref).max() <= tol and np.abs(f[0] - ref).max() <= tol
