"""Sampling at every width of the cluster kernel and at the ends of its range: one given byte, the full 256-byte window,
products of one and of several ring chunks, fewer heads than blocks and as many.  Sampled bytes equal the oracle's."""
import numpy as np
import pytest

from common import load_oracle, load_pkg, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,layers,given,new", [
    (128, 3, 1, 255),         # two heads, one row per warp
    (256, 2, 255, 1),         # a single draw at the end of the window
    (384, 2, 1, 60),
    (512, 4, 32, 224),
    (640, 2, 20, 30),
    (768, 1, 40, 24),
    (896, 2, 5, 20),          # odd chunk sizes
    (1024, 2, 16, 40),        # as many heads as blocks; the widest chunks
])
def test_every_width_against_oracle(hidden, layers, given, new):
    pkg, O = load_pkg(), load_oracle()
    kw = dict(hidden_dim=hidden, n_layers=layers, seq_len=256, population_size=8)
    cfg, ocfg, model, data = make_case(kw, data_len=20000, model_kind="random_all", model_seed=3)
    ctx = pkg.Context(cfg, 0, 2)
    ctx.upload_model(model)
    for seed, temp, mp, pen in ((5, 0.7, 0.05, 0.3), (6, 1.0, 0.0, 0.0)):
        want = O.generate(ocfg, model, data[:given], new, seed, temp, mp, pen)
        got = ctx.generate(data[:given], new, seed, temp, mp, pen)
        assert (got == want).all(), (seed, int((got != want).argmax()))
    ctx.close()


@pytest.mark.parametrize("hidden,seq_len,given,kw", [
    (128, 256, 12, {}), (128, 256, 13, {}),          # the last length that is decoded byte by byte, the first that is filled in one pass
    (384, 48, 47, {}), (512, 48, 18, {}),            # windows shorter than the cache
    (896, 256, 250, {}), (1024, 80, 64, {}),
    (256, 512, 200, dict(device_mask=15)), (256, 64, 30, dict(device_mask=15, device_gaussian=1)),
    (128, 64, 20, dict(shift_mlp_up=14)),            # a shift the evaluation's kernels do not take
])
def test_given_bytes_in_one_pass(hidden, seq_len, given, kw):
    """The cache that the evaluation kernels fill equals the one that decoding fills, also with overlays loaded."""
    pkg, O = load_pkg(), load_oracle()
    kw = dict(kw, hidden_dim=hidden, n_layers=2, seq_len=seq_len, population_size=8)
    cfg, ocfg, model, data = make_case(kw, data_len=20000, model_kind="random_all", model_seed=given)
    new = min(seq_len, 256) - given
    ctx = pkg.Context(cfg, 0, 2)
    ctx.upload_model(model)
    want = O.generate(ocfg, model, data[:given], new, 11, 0.8, 0.02, 0.3)
    assert (ctx.generate(data[:given], new, 11, 0.8, 0.02, 0.3) == want).all()
    ctx.upload_scales(np.random.RandomState(1).randint(-30, 90, pkg.scales_bytes(cfg)).astype(np.int8))
    assert (ctx.generate(data[:given], new, 11, 0.8, 0.02, 0.3) == want).all()
    ctx.close()
