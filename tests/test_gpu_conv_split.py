"""128-channel convolutions whose tiles leave SMs idle take two CTAs a tile
(k_conv_tc): the values are those of one CTA a tile."""
import numpy as np
import pytest

from test_surrogate import _rand_bf16, _taps

pytestmark = pytest.mark.gpu


# 76 images of 128 pixels are the last to be split on 152 SMs
@pytest.mark.parametrize("cin,taps,relu,resid", [(128, "enc5", True, True), (64, "enc5", True, False),
                                                 (128, "one", False, False)])
def test_split_tiles_give_the_same_values(engine_lib, cin, taps, relu, resid):
    import torch

    from tfm_gb300 import surrogate

    whole = torch.cuda.get_device_properties(0).multi_processor_count // 2 + 1
    rng = np.random.default_rng(cin)
    x = _rand_bf16(rng, (whole, 1, 128, cin))
    w = _rand_bf16(rng, (len(_taps(taps)), 128, cin), 0.05)
    bias = (rng.standard_normal(128) * 0.1).astype(np.float32)
    r = _rand_bf16(rng, (whole, 1, 128, 128)) if resid else None
    out, mask = surrogate.conv_bf16(x, w, _taps(taps), bias=bias, relu=relu, resid=r, want_mask=True)
    for n in (1, whole - 1):
        o, m = surrogate.conv_bf16(x[:n], w, _taps(taps), bias=bias, relu=relu,
                                   resid=None if r is None else r[:n], want_mask=True)
        assert np.array_equal(o, out[:n])
        assert np.array_equal(np.asarray(m).reshape(-1), np.asarray(mask).reshape(-1)[: np.asarray(m).size])
