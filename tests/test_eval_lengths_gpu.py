"""Evaluation at every form of the attention kernels (a warp per head at 16 and 32 tokens; tensor memory where a member has 64 to 512
rows in whole blocks of 32: two members or one in a tile, one to four tiles; for other lengths a warp per head up to 64 tokens, kept
scores up to 128, any length above), at ragged ends of their key blocks, and at row tiles that span members (lengths that are multiples
of 32 or padded to one), with and without overlays, against the CPU oracle: losses are equal."""
import numpy as np
import pytest

from common import load_oracle, load_pkg, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seq", [16, 32, 48, 64, 80, 96, 112, 128, 144, 160, 192, 224, 256, 272, 400, 512, 528])
@pytest.mark.parametrize("hidden", [128, 256, 384, 512, 640, 768, 896])
def test_losses_match_oracle(seq, hidden):
    if hidden > 128 and seq not in ((32, 80, 96, 128, 160) if hidden > 384 else (16, 32, 48, 64, 80, 96, 144, 224)):
        pytest.skip("covered at the smaller widths")
    pkg, O = load_pkg(), load_oracle()
    kw = dict(hidden_dim=hidden, n_layers=1, seq_len=seq, population_size=14, device_mask=15)
    cfg, ocfg, model, data = make_case(kw, data_len=9000, model_kind="random_all", model_seed=seq)
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ctx.set_dataset(data)
    ctx.eval_chunk(0xBEEF, 40, 2, 10)                       # a chunk that starts inside the population and fills no tile
    want = O.eval_losses(ocfg, model, data, 40, 0xBEEF, 2, 10)
    assert (ctx.read_losses(2, 10) == want).all()
    ctx.close()


@pytest.mark.parametrize("kw", [
    dict(hidden_dim=128, seq_len=48, shift_out=14), dict(hidden_dim=256, seq_len=128, shift_mlp_down=15, fixed_point=5),
    dict(hidden_dim=640, seq_len=32, fixed_point=6, sigma_shift=6),
    # rows that are not padded: the attention kernels that tensor memory takes no part in
    dict(hidden_dim=128, seq_len=80, shift_out=14), dict(hidden_dim=256, seq_len=112, shift_out=14),
    dict(hidden_dim=256, seq_len=144, shift_out=14), dict(hidden_dim=128, seq_len=400, shift_out=14),
])
def test_shifts_beyond_the_row_owning_form(kw):
    """Output shift plus rank-1 shift above 20: the two-kernel form at lengths and widths that otherwise never take it."""
    pkg, O = load_pkg(), load_oracle()
    kw = dict(kw, n_layers=1, population_size=8, device_mask=15)
    cfg, ocfg, model, data = make_case(kw, data_len=9000, model_kind="random_all", model_seed=1)
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ctx.set_dataset(data)
    assert ctx.fused_epilogues_active() == 0
    ctx.eval_chunk(0xBEEF, 40, 0, 8)
    assert (ctx.read_losses(0, 8) == O.eval_losses(ocfg, model, data, 40, 0xBEEF, 0, 8)).all()
    ctx.close()


@pytest.mark.parametrize("hidden,seq", [(128, 48), (256, 64), (384, 80), (512, 32), (640, 96), (768, 32), (896, 16), (1024, 64)])
def test_overlays_match_oracle(hidden, seq):
    pkg, O = load_pkg(), load_oracle()
    kw = dict(hidden_dim=hidden, n_layers=1, seq_len=seq, population_size=8, device_mask=15, chunk_relative_loss=1)
    cfg, ocfg, model, data = make_case(kw, data_len=5000, model_kind="random_all", model_seed=seq)
    scales = np.random.RandomState(hidden).randint(-30, 90, pkg.scales_bytes(cfg)).astype(np.int8)
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ctx.upload_scales(scales)
    ctx.set_dataset(data)
    ctx.eval_chunk(77, 16, 0, 8)
    want = O.eval_losses(ocfg, model, data, 16, 77, 0, 8, scales=scales)
    assert (ctx.read_losses(0, 8) == want).all()
    ctx.close()


@pytest.mark.parametrize("seq", [144, 256, 272, 512])
def test_flat_attention_matches_oracle(seq):
    """Every weight at its largest and every key alike (no query, one token): the attention sums reach the ends of their
    range."""
    pkg, O = load_pkg(), load_oracle()
    H = 128
    kw = dict(hidden_dim=H, n_layers=1, seq_len=seq, population_size=2, device_mask=0)
    cfg, ocfg, model, data = make_case(kw, data_len=3000, model_kind="random_all", model_seed=seq)
    wq = 256 * H + 3 * H + 2 * 4 * H * H + 5 * H + 2 * H
    model[wq:wq + H * H] = 0
    data[:] = 65
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ctx.set_dataset(data)
    ctx.eval_chunk(1, 0, 0, 2)
    assert (ctx.read_losses(0, 2) == O.eval_losses(ocfg, model, data, 0, 1, 0, 2)).all()
    ctx.close()


@pytest.mark.parametrize("kw,members", [
    (dict(hidden_dim=128, n_layers=2, seq_len=16, population_size=600), (0, 100, 256, 510, 512, 600)),
    (dict(hidden_dim=128, n_layers=1, seq_len=16, population_size=600, device_gaussian=1), (600,)),
    (dict(hidden_dim=128, n_layers=1, seq_len=16, population_size=600, vocab_size=768), (600,)),
    (dict(hidden_dim=128, n_layers=1, seq_len=16, population_size=600, chunk_relative_loss=1), (600,)),
])
def test_perturbations_of_few_and_many_pairs(kw, members):
    """Pairs hashed one by one and pairs filled from the shared noise table, on both sides of the count where the table
    starts; the last pairs reach its last rows."""
    pkg, O = load_pkg(), load_oracle()
    cfg, ocfg, model, data = make_case(dict(kw, device_mask=15), data_len=9000, model_kind="random_all", model_seed=9)
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ctx.set_dataset(data)
    pop = kw["population_size"]
    want = O.eval_losses(ocfg, model, data, 40, 0xFFFFFF00, 0, pop)          # the seeds wrap around
    for n in members:
        if n:
            ctx.eval_chunk(0xFFFFFF00, 40, pop - n, n)
            assert (ctx.read_losses(pop - n, n) == want[pop - n:]).all(), n
    ctx.close()


@pytest.mark.parametrize("hidden,seq,vocab,kind,scales", [
    (128, 16, 512, "random_all", False),        # tiles of four members, half a step of the row sums
    (256, 48, 768, "random", False), (384, 80, 1280, "random_all", True),
    (128, 272, 2816, "random_all", False),      # most logits saturate; several steps
    (1024, 32, 512, "random_all", True),        # the rank-1 shift on its own
    (128, 32, 1024, "flat", False),             # all logits alike: every byte zero
])
def test_wide_vocabulary_matches_oracle(hidden, seq, vocab, kind, scales):
    pkg, O = load_pkg(), load_oracle()
    kw = dict(hidden_dim=hidden, n_layers=1, seq_len=seq, population_size=10, device_mask=0 if kind == "flat" else 15, vocab_size=vocab,
              chunk_relative_loss=int(scales))
    cfg, ocfg, model, data = make_case(kw, data_len=6000, model_kind="random" if kind == "flat" else kind, model_seed=vocab)
    if kind == "flat":
        model[:vocab * hidden] = 1
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ov = None
    if scales:
        ov = np.random.RandomState(hidden).randint(-30, 90, pkg.scales_bytes(cfg)).astype(np.int8)
        ctx.upload_scales(ov)
    ctx.set_dataset(data)
    ctx.eval_chunk(5, 11, 0, 10)
    assert (ctx.read_losses(0, 10) == O.eval_losses(ocfg, model, data, 11, 5, 0, 10, scales=ov)).all()
    ctx.close()


@pytest.mark.parametrize("hidden,seq", [(256, 128), (384, 128), (512, 128), (256, 32), (384, 96), (512, 80), (128, 128)])
def test_few_and_many_tiles_match_oracle(hidden, seq):
    """Chunks of 18, 20, 74, 76 and 320 tiles of 128 rows: around the counts from which a tile has one block instead of two and
    the widest column tiles.  The first and the last members of each chunk are compared."""
    pkg, O = load_pkg(), load_oracle()
    pop = 320 * 128 // seq // 2 * 2
    kw = dict(hidden_dim=hidden, n_layers=1, seq_len=seq, population_size=pop, device_mask=15)
    cfg, ocfg, model, data = make_case(kw, data_len=9000, model_kind="random_all", model_seed=seq)
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ctx.set_dataset(data)
    for tiles in (18, 20, 74, 76, 320):
        n = tiles * 128 // seq // 2 * 2
        ctx.eval_chunk(0xBEEF, 40, 0, n)
        got = ctx.read_losses(0, n)
        for at in (0, n - 6):
            assert (got[at:at + 6] == O.eval_losses(ocfg, model, data, 40, 0xBEEF, at, 6)).all(), (tiles, at)
    ctx.close()
