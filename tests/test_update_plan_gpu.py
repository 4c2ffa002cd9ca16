"""The whole-model update (one noise table, written operands, batched vote GEMM) against the CPU oracle where its
alignment and dispatch can go wrong: populations below and just above a contraction block, widths that are odd multiples of
128 (half-filled vote tiles), Gaussian noise, fitness beyond -1..1 (the general operand path), a wide vocabulary.  Weights,
counts and the fp32 state are equal bit for bit."""
import numpy as np
import pytest

from common import load_oracle, load_pkg, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,amp", [
    (dict(hidden_dim=128, n_layers=1, seq_len=16, population_size=2), 1),              # a single pair
    (dict(hidden_dim=128, n_layers=3, seq_len=16, population_size=226), 1),            # 113 pairs: 113 + 15 columns fill one block exactly
    (dict(hidden_dim=384, n_layers=2, seq_len=16, population_size=228), 1),            # one more spills into a second block
    (dict(hidden_dim=256, n_layers=2, seq_len=16, population_size=1002, device_gaussian=1, device_mask=15), 1),
    (dict(hidden_dim=256, n_layers=1, seq_len=16, population_size=514, device_mask=3), 42),   # 42 * 3 <= 127
    (dict(hidden_dim=128, n_layers=1, seq_len=16, population_size=66, vocab_size=1024), 1),
    (dict(hidden_dim=640, n_layers=1, seq_len=16, population_size=600, device_mask=3), 1),
])
def test_update_against_oracle(kw, amp):
    pkg, O = load_pkg(), load_oracle()
    cfg, ocfg, model, data = make_case(kw, data_len=4000, model_kind="random_all", model_seed=9)
    pairs = kw["population_size"] // 2
    rng = np.random.RandomState(4)
    opt = np.zeros(O.opt_bytes(ocfg), np.uint8)
    ctx = pkg.Context(cfg, 0, 2)
    ctx.upload_model(model)
    for step in range(3):
        fit = rng.randint(-amp, amp + 1, pairs).astype(np.int32)
        ctx.write_fitness(fit)
        n = ctx.apply_update(0xFFFFFF00 + 97 * step, 0.4)          # seeds wrap around 2^32
        assert n == O.update(ocfg, model, opt, fit, (0xFFFFFF00 + 97 * step) & 0xFFFFFFFF, 0.4)
        assert (ctx.download_model() == model).all(), step
        assert (ctx.download_opt_state() == opt).all(), step
    ctx.close()


@pytest.mark.parametrize("amp,kw", [
    (8, dict(device_mask=15)),                                     # 120: still inside a byte
    (9, dict(device_mask=15)),                                     # 135: the first that wraps
    (127, dict(device_mask=1, device_gaussian=1)),                 # sums of three noise values
    (200, dict(device_mask=3, vocab_size=768)),                    # beyond int8 itself, more outputs than four widths
    (100000, dict(device_mask=15)),
])
def test_products_that_wrap_equal_the_isolated_update(amp, kw):
    """Fitness times noise beyond a byte wraps on the outputs' side whatever the matrix's shape: every matrix of the model
    update equals the isolated update of that matrix, which has no other form.  Vectors do not wrap: they equal the oracle's."""
    import torch
    pkg, O = load_pkg(), load_oracle()
    H, V = 128, kw.get("vocab_size", 256)
    pop = 614
    cfg = pkg.default_config(hidden_dim=H, n_layers=1, seq_len=16, population_size=pop, **kw)
    ctx = pkg.Context(cfg, 0, 2)
    rng = np.random.RandomState(amp)
    model = rng.randint(-127, 128, pkg.model_bytes(cfg)).astype(np.int8)
    fit = rng.randint(-amp, amp + 1, pop // 2).astype(np.int32)
    ctx.upload_model(model)
    ctx.write_fitness(fit)
    ctx.apply_update(77, 0.4)
    got, state = ctx.download_model(), ctx.download_opt_state().view(np.float32).reshape(-1, 3)
    after_init = V * H + 3 * H + 4 * H * H + 4 * H + 4 * H * H + H
    w_q = after_init + 2 * H
    w_up = w_q + 4 * H * H + 2 * H
    w_down = w_up + 4 * H * H + 4 * H
    ocfg = O.make_config(hidden_dim=H, n_layers=1, seq_len=16, population_size=pop, **kw)
    want, want_state = model.copy(), np.zeros(O.opt_bytes(ocfg), np.uint8)
    O.update(ocfg, want, want_state, fit, 77, 0.4)
    want_state = want_state.view(np.float32).reshape(-1, 3)
    for off, length in ((V * H, 3 * H), (V * H + 3 * H + 4 * H * H, 4 * H), (after_init - H, 3 * H), (w_up - 2 * H, 2 * H), (w_down - 4 * H, 4 * H),
                        (w_down + 4 * H * H, 3 * H)):
        assert (state[off:off + length] == want_state[off:off + length]).all() and (got[off:off + length] == want[off:off + length]).all(), off
    d_fit = torch.from_numpy(fit).cuda()
    for off, rows, cols, a, b in ((0, H, V, 0, H), (V * H + 3 * H, H, 4 * H, 510, 511), (V * H + 3 * H + 4 * H * H + 4 * H, 4 * H, H, 512, 513),
                                  (w_q, H, H, 200, 201), (w_up, H, 4 * H, 400, 401), (w_down, 4 * H, H, 402, 403)):
        w = torch.from_numpy(model[off:off + rows * cols].copy()).cuda()
        opt = torch.zeros(rows * cols, 3, device="cuda")
        torch.cuda.synchronize()
        ctx.update_matrix(w.data_ptr(), opt.data_ptr(), rows, cols, a, b, 0, d_fit.data_ptr(), pop // 2, 77, 0.4, 0, False)
        assert (opt.cpu().numpy() == state[off:off + rows * cols]).all(), (rows, cols, a)
        assert (w.cpu().numpy() == got[off:off + rows * cols]).all(), (rows, cols, a)
    ctx.close()
