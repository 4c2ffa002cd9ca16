"""Products that pairs of thread blocks form together (cta_group::2): the same losses as the same members in chunks too small for pairs,
as the two-kernel form, for every member, and as the CPU oracle for the members of the first and the last row tile.  The sizes: an odd number
of row tiles (the last pair forms one twice and stores it once) where tiles hold several members -- tiles of one member come in even
numbers, as members do --, sub-tiles of 256 and of 128 columns, one and several of them, clusters of four (a pair for each half of the columns),
even and uneven halves.  That these sizes do take pairs is asked in test_host_paths_cpu.py."""
import numpy as np
import pytest

from common import cfg_pair, load_oracle, load_pkg, make_case

pytestmark = pytest.mark.gpu

SEED = 0x00C0FFEE


EVALUATIONS = [                # hidden, layers, seq, pop, other settings
    (384, 2, 64, 594, {}),     # K 1536, 297 row tiles of two members each; three sub-tiles of 128; two layers: three and one dots follow
    (512, 1, 128, 298, {}),    # K 2048, tiles of one member, two sub-tiles of 256
    (512, 1, 128, 298, dict(fixed_point=5, sigma_shift=4)),          # the output projection's shifts apart
    (512, 1, 96, 396, {}),     # 297 tiles across members of 96 rows
    (256, 1, 128, 100, {}),    # Q|K|V alone, one sub-tile a unit
    (640, 1, 64, 594, {}),     # clusters of four, 384 + 256 columns
    (1024, 1, 128, 298, {}),   # clusters of four, 512 + 512 columns; K 1024 in the up projection, too
]


def small_chunk(hidden, seq):
    """The most members whose products are too few tiles for pairs: MLP-up below 4 x 148, Q|K|V below 2 x 148."""
    return min(4 * 148 * 256 // (4 * hidden) - 1, 2 * 148 // 3 - 1) * 128 // seq & ~1


@pytest.mark.parametrize("hidden,layers,seq,pop,other", EVALUATIONS)
def test_pairs_equal_single_blocks_and_oracle(hidden, layers, seq, pop, other):
    pkg, O = load_pkg(), load_oracle()
    kw = dict(hidden_dim=hidden, n_layers=layers, seq_len=seq, population_size=pop, device_mask=3, **other)
    cfg, ocfg, model, data = make_case(kw, data_len=60000, model_kind="random_all")

    def losses(level, chunk=pop):
        ctx = pkg.Context(cfg, 0, pop)
        ctx.set_fused_epilogues(level)
        ctx.upload_model(model)
        ctx.set_dataset(data)
        for first in range(0, pop, chunk):
            ctx.eval_chunk(SEED + 5, seq, first, min(chunk, pop - first))
        out = ctx.read_losses(0, pop)
        ctx.close()
        return out

    got = losses(2)
    assert (got == losses(2, small_chunk(hidden, seq))).all()
    assert (got == losses(0)).all()
    for first in (0, pop - 4):
        assert (got[first:first + 4] == O.eval_losses(ocfg, model, data, seq, SEED + 5, first, 4)).all(), first


MODEL_UPDATES = [              # hidden, layers, pairs, pairs of blocks
    (256, 2, 1300, True),      # 11 blocks of the contraction in several splits
    (384, 1, 1501, True),      # three tiles of 128 outputs: the second half of the last pair's tile is not stored
    (640, 1, 370, True),       # five; the shortest contraction
    (640, 1, 300, False),      # single blocks
]


@pytest.mark.parametrize("hidden,layers,pairs", [u[:3] for u in MODEL_UPDATES])
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


RECONSTRUCTIONS = [            # rows, cols, pairs, pairs of blocks
    (2048, 2560, 1000, True),  # 160 tiles
    (2048, 2688, 1000, False), # 21 row tiles of outputs: single blocks
    (2048, 2560, 500, False),  # a short contraction
    (512, 1024, 2000, False),  # 16 tiles: too few
    (512, 1152, 2000, False),
]


@pytest.mark.parametrize("rows,cols,pairs", [r[:3] for r in RECONSTRUCTIONS])
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


MATRIX_UPDATES = [             # rows, cols, pairs, int8 fitness
    (1024, 1024, 16384, False),          # 32 tiles in 10 parts of the contraction, of 13 blocks, the last of 11
    (1024, 1280, 10000, True),           # 40 tiles in 8 parts of 20 blocks, the last of 18
]


@pytest.mark.parametrize("rows,cols,pairs,int8fit", MATRIX_UPDATES)
def test_matrix_update_of_pairs_with_a_split_contraction(rows, cols, pairs, int8fit):
    import torch
    pkg, O = load_pkg(), load_oracle()
    cfg, ocfg = cfg_pair(device_mask=3, population_size=2 * pairs)
    rng = np.random.default_rng(rows + int8fit)
    w0 = rng.integers(-127, 128, rows * cols).astype(np.int8)
    fit = (rng.integers(-127, 128, pairs) if int8fit else rng.integers(-1, 2, pairs)).astype(np.int32)
    ctx = pkg.Context(cfg, 0, 2)
    d_w, d_st, d_fit = torch.from_numpy(w0.copy()).cuda(), torch.zeros(rows * cols * 3, dtype=torch.float32, device="cuda"), torch.from_numpy(fit).cuda()
    torch.cuda.synchronize()
    n = ctx.update_matrix(d_w.data_ptr(), d_st.data_ptr(), rows, cols, 402, 403, 1000, d_fit.data_ptr(), pairs, 2, 2.5, optimizer=0, split=int8fit)
    ctx.close()
    w1, st1 = d_w.cpu().numpy(), d_st.cpu().numpy().reshape(-1, 3)
    assert n == (w1 != w0).sum() > 0
    k, n_list = np.arange(rows), np.arange(0, cols, 37).astype(np.int32)
    for col, votes in zip(n_list, O.vote_columns(ocfg, fit, rows, 402, 403, 1000, 2, n_list)):
        idx = ((k >> 2) * cols + col) * 4 + (k & 3)                 # packed order [k/4][n][4]
        w, st = w0[idx].copy(), np.zeros((rows, 3), np.float32)
        O.adam_from_votes(ocfg, w, st, votes, 2.5)
        assert (w1[idx] == w).all() and (st1[idx].view(np.uint32) == st.view(np.uint32)).all(), col


PROJECTIONS = [(37 * 128, 1024, 4096), (37 * 128 - 64, 1024, 4096)]          # rows, K, N: an odd number of row tiles, the last one whole and half


@pytest.mark.parametrize("rows,k,n", PROJECTIONS)
def test_projection_of_pairs_with_an_odd_row_tile(rows, k, n):
    """Beside the transposed epilogue, which results at an odd word take and whose blocks work alone, for every row; the first and the last
    pair of members beside the oracle; nothing is stored outside."""
    import torch
    pkg, O = load_pkg(), load_oracle()
    cfg, ocfg = cfg_pair(device_mask=3, population_size=64)
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    x = torch.clamp(torch.round(torch.randn((rows, k), generator=g, device="cuda") * 32.0), -127, 127).to(torch.int8)
    w = torch.randint(-127, 128, (k * n,), generator=g, device="cuda", dtype=torch.int8)
    out = torch.full((2, rows * n + 128 * n), 99, dtype=torch.int8, device="cuda")
    ctx = pkg.Context(cfg, 0, 2)
    torch.cuda.synchronize()
    for o, offset in zip(out, (64, 68)):
        ctx.perturbed_projection(x.data_ptr(), w.data_ptr(), o.data_ptr() + offset, rows, k, n, 32, 7, 200, 201, 7, 8, on_device=True)
    ctx.close()
    y, z = (o[f:f + rows * n].view(rows, n) for o, f in zip(out, (64, 68)))
    assert torch.equal(y, z)
    for o, f in zip(out, (64, 68)):
        assert (o[:f] == 99).all() and (o[f + rows * n:] == 99).all()
    xs, ws = x.cpu().numpy(), w.cpu().numpy()
    for j in (0, rows // 64 - 1):
        assert (y[64 * j:64 * j + 64].cpu().numpy() == O.projection(ocfg, xs[64 * j:64 * j + 64], ws, k, n, 32, 7 + j, 200, 201, 7, 8)).all(), j


NEWTON_SCHULZ = [(512, 896, True), (640, 1024, False), (1024, 1024, True), (2304, 2304, True)]          # rows, cols, pairs of blocks


@pytest.mark.parametrize("rows,cols", [n[:2] for n in NEWTON_SCHULZ])
def test_newton_schulz_in_pairs(rows, cols):
    """Pairs of tiles in both products; an odd number of row tiles (single blocks); a square matrix; 90 pairs in the Gram matrix and 162 in the
    step, more than fit at once, so that a pair goes on to another item, also after a tile below the diagonal."""
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
