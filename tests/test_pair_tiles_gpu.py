"""Products that pairs of thread blocks form together (cta_group::2): the same losses as the two-kernel form, whose blocks work alone, for
every member, and as the CPU oracle for the members of the first and the last row tile.  The sizes: an odd number of row tiles (the last
pair forms one twice and stores it once), tiles of one member and of several, sub-tiles of 256 and of 128 columns, clusters of four
(a pair for each half of the columns), even and uneven halves."""
import numpy as np
import pytest

from common import cfg_pair, load_oracle, load_pkg, make_case

pytestmark = pytest.mark.gpu

SEED = 0x00C0FFEE


@pytest.mark.parametrize("hidden,layers,seq,pop", [
    (384, 2, 64, 594),         # K 1536, 297 row tiles of two members each; three sub-tiles of 128; two layers: three and one dots follow
    (512, 1, 128, 298),        # K 2048, tiles of one member, two sub-tiles of 256
    (512, 1, 96, 396),         # 297 tiles across members of 96 rows
    (640, 1, 64, 594),         # clusters of four, 384 + 256 columns
    (1024, 1, 128, 298),       # clusters of four, 512 + 512 columns; K 1024 in the up projection, too
])
def test_pairs_equal_single_blocks_and_oracle(hidden, layers, seq, pop):
    pkg, O = load_pkg(), load_oracle()
    kw = dict(hidden_dim=hidden, n_layers=layers, seq_len=seq, population_size=pop, device_mask=3)
    cfg, ocfg, model, data = make_case(kw, data_len=60000, model_kind="random_all")

    def losses(level):
        ctx = pkg.Context(cfg, 0, pop)
        ctx.set_fused_epilogues(level)
        ctx.upload_model(model)
        ctx.set_dataset(data)
        ctx.eval_chunk(SEED + 5, seq, 0, pop)
        out = ctx.read_losses(0, pop)
        ctx.close()
        return out

    got = losses(2)
    assert (got == losses(0)).all()
    for first in (0, pop - 4):
        assert (got[first:first + 4] == O.eval_losses(ocfg, model, data, seq, SEED + 5, first, 4)).all(), first


@pytest.mark.parametrize("hidden,layers,pairs", [
    (256, 2, 1300),            # 11 blocks of the contraction in several splits
    (384, 1, 1501),            # three tiles of 128 outputs: the second half of the last pair's tile is not stored
    (640, 1, 300),             # five; contraction of three blocks
])
def test_vote_tiles_of_pairs(hidden, layers, pairs):
    pkg, O = load_pkg(), load_oracle()
    kw = dict(hidden_dim=hidden, n_layers=layers, seq_len=16, population_size=2 * pairs, device_mask=15)
    cfg, ocfg, model, data = make_case(kw, data_len=4000, model_kind="random_all", model_seed=3)
    opt = np.zeros(O.opt_bytes(ocfg), np.uint8)
    ctx = pkg.Context(cfg, 0, 2)
    ctx.upload_model(model)
    fit = np.random.RandomState(hidden).randint(-1, 2, pairs).astype(np.int32)
    ctx.write_fitness(fit)
    assert ctx.apply_update(SEED, 0.4) == O.update(ocfg, model, opt, fit, SEED, 0.4)
    assert (ctx.download_model() == model).all()
    assert (ctx.download_opt_state() == opt).all()
    ctx.close()


@pytest.mark.parametrize("rows,cols,pairs", [
    (512, 1024, 2000),         # tiles and splits of the contraction enough for pairs
    (512, 1152, 2000),         # nine row tiles of outputs: single blocks
])
def test_isolated_votes_of_pairs(rows, cols, pairs):
    import torch
    pkg, O = load_pkg(), load_oracle()
    cfg, ocfg = cfg_pair(device_mask=3, population_size=2 * pairs)
    fit = np.random.RandomState(rows + cols).randint(-1, 2, pairs).astype(np.int32)
    ctx = pkg.Context(cfg, 0, 2)
    d_fit, votes = torch.from_numpy(fit).cuda(), torch.zeros(rows * cols, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.update_reconstruct(d_fit.data_ptr(), pairs, rows, cols, 402, 403, 1000, 2, votes.data_ptr(), on_device=True)
    ctx.close()
    n_list = np.arange(0, cols, 37).astype(np.int32)
    got = votes.cpu().numpy().reshape(rows // 4, cols, 4)[:, n_list, :].transpose(1, 0, 2).reshape(len(n_list), rows)      # packed order [k/4][n][4]
    assert (got == O.vote_columns(ocfg, fit, rows, 402, 403, 1000, 2, n_list)).all()


@pytest.mark.parametrize("rows,cols", [(512, 896), (640, 1024), (1024, 1024)])
def test_newton_schulz_in_pairs(rows, cols):
    """Pairs of tiles in both products; an odd number of row tiles (single blocks); more pairs than fit at once in the Gram matrix."""
    from test_muon_gpu import test_newton_schulz_against_float64 as check
    check(rows, cols)


@pytest.mark.parametrize("seq", [32, 48, 16])          # a warp's own tables, padded to 64 rows, tables of the tile
def test_logits_of_short_windows(seq):
    pkg, O = load_pkg(), load_oracle()
    kw = dict(hidden_dim=128, n_layers=1, seq_len=seq, vocab_size=512, population_size=22, device_mask=15)
    cfg, ocfg, model, data = make_case(kw, data_len=60000, model_kind="random_all")
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ctx.set_dataset(data)
    ctx.eval_chunk(SEED + 2, 5, 0, 22)
    assert (ctx.read_losses(0, 22) == O.eval_losses(ocfg, model, data, 5, SEED + 2, 0, 22)).all()
    ctx.close()
