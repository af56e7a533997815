"""The 3x3, 64-channel convolution that reads every input row once
(k_conv_rows) at the sizes where its runs, its accumulator ring and its window
ring end, and its repeatability."""
import numpy as np
import pytest

from test_surrogate import _rand_bf16, _ref_conv

pytestmark = pytest.mark.gpu


# one row; fewer rows than the dilation; rows not a multiple of it; runs that
# are cut between CTAs (more rows than SMs), up and down; unequal steps
@pytest.mark.parametrize("B,H,W,dh,dw", [(1, 1, 128, 1, 1), (1, 3, 128, 8, 8), (2, 7, 128, 3, 3),
                                         (3, 131, 128, -2, -2), (1, 77, 384, 5, -4), (2, 200, 256, -1, 8)])
def test_conv_rows_matches_oracle(engine_lib, B, H, W, dh, dw):
    from tfm_gb300 import surrogate

    taps = [(r * dh, c * dw) for r in (-1, 0, 1) for c in (-1, 0, 1)]
    rng = np.random.default_rng(B * 1000 + H)
    x = _rand_bf16(rng, (B, H, W, 64))
    w = _rand_bf16(rng, (9, 64, 64), 1.0 / 24)
    bias = (rng.standard_normal(64) * 0.1).astype(np.float32)
    resid = _rand_bf16(rng, (B, H, W, 64))
    out, mask = surrogate.conv_bf16(x, w, taps, bias=bias, relu=True, resid=resid, want_mask=True)
    pre, ref = _ref_conv(x, w, taps, bias, True, resid)
    err = np.abs(surrogate.from_bf16(out) -
                 surrogate.from_bf16(surrogate.to_bf16(ref.astype(np.float32))).astype(np.float64))
    # one BF16 step of the value, and the FP32 sum's rounding where it cancels
    step = 2.0 ** (np.floor(np.log2(np.maximum(np.abs(ref), 1e-30))) - 7)
    assert np.all(err <= step + 2e-5)
    assert np.count_nonzero(err) <= 0.01 * err.size
    bits = np.unpackbits(mask.view(np.uint8), bitorder="little").reshape(pre.shape).astype(bool)
    assert np.all(np.abs(pre[bits != (pre > 0)]) < 1e-5)


def test_predictions_repeat_bit_for_bit(engine_lib):
    """Every wait of the pipeline guards a buffer that is written again: a
    missing one shows as a value that differs between passes."""
    from tfm_gb300 import surrogate

    types, lad, _ = surrogate.make_sequences(32, 1024, 5)
    with surrogate.Surrogate("batch 32\n", seed=4) as net:
        p = net.params()
        p[-65:-1] = np.random.default_rng(3).standard_normal(64) * 0.1
        net.set_params(p)
        first = net.predict(types, lad)
        for _ in range(60):
            assert np.array_equal(net.predict(types, lad), first)
        assert net.error_flags() == 0


# as above for the weight gradients; the last two take the kernel that copies
# the input once a tap (column steps to the left, images of 64-pixel blocks)
@pytest.mark.parametrize("B,H,W,dh,dw", [(1, 1, 128, 1, 1), (1, 2, 128, 8, 8), (2, 7, 128, 3, 3),
                                         (3, 131, 128, -2, 2), (1, 77, 384, 5, 4), (2, 200, 256, -1, 8),
                                         (1, 9, 128, 2, -2), (1, 9, 192, 2, 2)])
def test_wgrad_rows_matches_oracle(engine_lib, B, H, W, dh, dw):
    from tfm_gb300 import surrogate

    taps = [(r * dh, c * dw) for r in (-1, 0, 1) for c in (-1, 0, 1)]
    rng = np.random.default_rng(B * 1000 + H + W)
    x = _rand_bf16(rng, (B, H, W, 64))
    dy = _rand_bf16(rng, (B, H, W, 64))
    dwt, db = surrogate.wgrad_bf16(x, dy, taps)
    xf = surrogate.from_bf16(x).astype(np.float64)
    yf = surrogate.from_bf16(dy).astype(np.float64)
    ref = np.zeros((9, 64, 64))
    for t, (a, b) in enumerate(taps):
        sh = np.zeros_like(xf)
        h0, h1, w0, w1 = max(0, -a), min(H, H - a), max(0, -b), min(W, W - b)
        if h0 < h1 and w0 < w1:
            sh[:, h0:h1, w0:w1] = xf[:, h0 + a:h1 + a, w0 + b:w1 + b]
        ref[t] = np.tensordot(yf, sh, axes=([0, 1, 2], [0, 1, 2]))
    # FP32 sums over up to 1e5 pixels, against the largest entry
    assert np.abs(dwt - ref).max() <= 1e-4 * np.abs(ref).max()
    refb = yf.sum(axis=(0, 1, 2))
    assert np.abs(db - refb).max() <= 1e-4 * np.abs(refb).max()
    assert np.array_equal(surrogate.wgrad_bf16(x, dy, taps)[0], dwt)
