"""What the counting sort refuses, the bucket path refuses too, where no bucket
overflows: sort cells wider than the buckets, and a sort cell whose beads
spread over the eight buckets around a corner."""
import numpy as np
import pytest

from helpers import baseline_params, ccp_params

pytestmark = pytest.mark.gpu


def _sims(text, preset):
    from tfm_gb300.ccpgpu import ChrSim

    kernel = "pair_kernel 2\n" if preset == "ccp" else "pair_kernel 4\n"
    for extra in ("", kernel):
        yield ChrSim(text + extra, seed=3)


def _refuses(h):
    from tfm_gb300.ccpgpu import CcpError

    h.error_flags(clear=True)
    for _ in range(2):
        with pytest.raises(CcpError, match="cell list"):
            h.forces()
        h.error_flags(clear=True)
    with pytest.raises(CcpError):
        h.run_steps(1)


@pytest.mark.parametrize("preset", ["ccp", "baseline"])
def test_wide_sort_cells(engine_lib, preset):
    """Contact cutoff 12: sort cells of side 6, buckets of 2 or 2.5."""
    n = 600
    text = "force_field %s\nnumber_of_particles %d\nnucleus_radius 15\ncontact_cutoff 12\n" % (preset, n)
    k = np.arange(300)
    x = np.concatenate([0.2 + 0.82 * np.stack([k % 7, k // 7 % 7, k // 49], 1),
                        -0.2 - 0.82 * np.stack([k % 7, k // 7 % 7, k // 49], 1)]).astype(np.float32)
    for h in _sims(text, preset):
        assert h.system_info(0).cell_side == 6.0
        h.set_types(np.zeros(n, np.int32))
        h.set_positions(x)
        _refuses(h)


@pytest.mark.parametrize("preset", ["ccp", "baseline"])
def test_sort_cell_over_eight_buckets(engine_lib, preset):
    """256 beads of one sort cell, 32 in each of the eight buckets that meet
    in it: a bucket's corner (a multiple of the largest cutoff x 1.0001) lies
    next to the lower corner of that cell."""
    n = 600
    rc = 2.0 if preset == "ccp" else 2.5
    text = ccp_params(n, cvf=0.02)[0] if preset == "ccp" else baseline_params(n, "nucleus_radius 15\n")
    k = np.arange(256)
    octant = np.stack([k >> 5 & 1, k >> 6 & 1, k >> 7], 1)
    t = np.stack([k % 4, k // 4 % 4, k // 16 % 2], 1) / 4.0
    # below the corner: 2e-5 .. 1.2e-4 of the 2e-4 left; above it: 0.1 .. 0.8
    x = np.zeros((n, 3))
    x[:256] = rc + np.where(octant == 0, 2e-5 + 1e-4 * t, 0.1 + 0.7 * t)
    j = np.arange(n - 256)
    x[256:] = -0.3 - 0.9 * np.stack([j % 7, j // 7 % 7, j // 49], 1)
    for h in _sims(text, preset):
        side = h.system_info(0).cell_side
        assert (np.floor(x[:256].astype(np.float32) / side) == 2).all() and side == rc / 2
        h.set_types(np.zeros(n, np.int32))
        h.set_positions(x.astype(np.float32))
        _refuses(h)
