"""Gradients of the pair features and of the distance embedding (k_pair_bwd) at
the smallest network, and at one with another map size and an odd batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins,batch", [(128, 1), (256, 3)])
def test_pair_gradients_match_oracle(engine_lib, bins, batch):
    from oracle import surrogate_oracle as so
    from tfm_gb300 import surrogate

    text = ("seq_len %d\nbins %d\nbatch %d\nenc_layers 1\nhead_layers 1\ndilations 1\n"
            % (bins, bins, batch))
    rng = np.random.default_rng(bins)
    types, lad, _ = surrogate.make_sequences(batch, bins, 3)
    i = np.arange(bins)
    maps = 0.5 / (1.0 + np.abs(i[:, None] - i[None, :])) ** 1.2 * (1.0 + 0.2 * rng.random((batch, bins, bins)))
    maps = (0.5 * (maps + maps.transpose(0, 2, 1))).astype(np.float32)
    rows = np.arange(batch, dtype=np.int32)[::-1].copy()
    with surrogate.Surrogate(text, seed=2) as net:
        p = net.params()
        p[-65:-1] = rng.standard_normal(64) * 0.5
        net.set_params(p)
        net.set_dataset(types, lad, maps)
        p = net.params()  # the dataset sets the output bias
        net.loss_grad(rows)
        g = net.grads()
        assert net.error_flags() == 0
    cfg = so.config(seq_len=bins, bins=bins, enc_layers=1, head_layers=1, dilations=(1,))
    _, gref = so.loss_and_grads(p.astype(np.float64), cfg, types[rows], lad[rows], maps[rows], maps)
    off = 0
    for name, shape in so.layout(cfg):
        n = int(np.prod(shape))
        a, b = g[off:off + n].astype(np.float64), gref[off:off + n]
        off += n
        if name in ("E", "proj.W", "proj.b"):
            # du and dv are rounded to BF16 (2^-9 relative) and pass one BF16
            # matrix product; the masks of a few pixels at zero may differ
            assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b), name
            assert a @ b >= 0.999 * np.linalg.norm(a) * np.linalg.norm(b), name
