"""Pairs within a rounding of the Lennard-Jones cutoff count on every path or on
none: FP32 forms of d^2 that differ in the last bit fall on either side."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(n):
    """Pair positions whose d^2 = 6.25 depends on the order of its FP32 sum."""
    rng = np.random.default_rng(0)
    out = []
    while len(out) < n:
        u = rng.standard_normal((4096, 3))
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        c = rng.uniform(-0.3, 0.3, (4096, 3))
        a, b = (c - 1.25 * u).astype(np.float32), (c + 1.25 * u).astype(np.float32)
        d = (a - b).astype(np.float64)  # exact
        f32 = np.float32
        forms = [((d[:, k] ** 2).astype(f32) + d[:, i] ** 2).astype(f32) + d[:, j] ** 2
                 for i, j, k in ((0, 2, 1), (1, 2, 0), (1, 0, 2))]
        side = [f.astype(f32) <= f32(6.25) for f in forms]
        mixed = (side[0] != side[1]) | (side[0] != side[2])
        out += list(zip(a[mixed], b[mixed]))
    return out[:n]


# 32, 16 and 8 lanes a bead on the bucket path; persistent; the other kernels
@pytest.mark.parametrize("systems", [400, 1600, 3200])
def test_pairs_at_the_cutoff(engine_lib, systems):
    from tfm_gb300.ccpgpu import Batch

    x = np.zeros((systems, 3, 3), np.float32)
    for k, (a, b) in enumerate(_pairs(systems)):
        x[k, 0], x[k, 2] = a, b
        # a B bead between them in the chain, out of its shorter reach of both
        v = np.cross(b - a, [0.31, 0.52, 0.79])
        x[k, 1] = 1.4 * v / np.linalg.norm(v) * (1.0 if v[0] > 0 else -1.0)
    types = np.tile(np.array([0, 1, 0], np.int32), systems)
    ref = None
    for text in ("pair_kernel 4\n", "", "persistent 1\n", "pair_kernel 4\npair_lanes 1\n",
                 "pair_kernel 2\n", "pair_kernel 0\n", "pair_kernel 1\n", "pair_kernel 3\n"):
        h = Batch("force_field baseline\ncontact_bins 2\nnumber_of_lbs 0\n" + text, [3] * systems,
                  n_chains=[3] * systems, radii=[2.45] * systems, seeds=list(range(systems)))
        h.set_types(types)
        h.set_positions(x.reshape(-1, 3))
        k0 = h.kernel_count()
        f = h.forces()
        if text == "":
            assert h.kernel_count() - k0 == 2  # the buckets and their force kernel
        ref = f if ref is None else ref
        # wall forces of some 100 kT/sigma in FP32; the pair's jump is 0.0195
        assert np.abs(f - ref).max() < 5e-3
        h.close()
