"""Attention in tensor memory at score shifts other than the default, at weight tables from one-hot (every row divides by a single
weight, exact quotients) to nearly flat, and at the widest weights, in windows of one to four tiles with ragged ends, and in chunks
whose blocks take several heads after one another, against the CPU oracle: losses are equal."""
import pytest

from common import load_oracle, load_pkg, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seq,kw", [
    (48, dict(shift_attn=5, softmax_exp_scale=1.0)), (64, dict(softmax_exp_scale=0.3)), (96, dict(shift_attn=12)), (128, dict(softmax_scale_bit=20, softmax_exp_scale=200.0)),
    (160, dict(shift_attn=7, softmax_exp_scale=30.0)), (256, dict(softmax_exp_scale=0.3)), (288, dict(shift_attn=21)), (400, dict(shift_attn=0, softmax_scale_bit=3)),
    (512, dict(softmax_scale_bit=20, softmax_exp_scale=500.0)),
])
def test_losses_match_oracle(seq, kw):
    pkg, O = load_pkg(), load_oracle()
    kw = dict(kw, hidden_dim=128, n_layers=1, seq_len=seq, population_size=10, device_mask=15)
    cfg, ocfg, model, data = make_case(kw, data_len=9000, model_kind="random_all", model_seed=seq)
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ctx.set_dataset(data)
    ctx.eval_chunk(0xBEEF, 40, 0, 10)
    assert (ctx.read_losses(0, 10) == O.eval_losses(ocfg, model, data, 40, 0xBEEF, 0, 10)).all()
    ctx.close()


@pytest.mark.parametrize("seq,members", [(48, 352), (64, 352), (256, 128), (288, 120), (512, 80)])
def test_blocks_that_take_several_heads(seq, members):
    """Items of one or two members' heads, at least two for every stage of a block's ring (4, 3 or 2 stages by length, 148 SMs) and a ragged
    last round: stages are filled again, barriers go through both parities.  Members of the first, a middle and the last round are compared."""
    pkg, O = load_pkg(), load_oracle()
    kw = dict(hidden_dim=512, n_layers=1, seq_len=seq, population_size=members, device_mask=15)
    cfg, ocfg, model, data = make_case(kw, data_len=9000, model_kind="random_all", model_seed=seq)
    ctx = pkg.Context(cfg, 0, 0)
    ctx.upload_model(model)
    ctx.set_dataset(data)
    ctx.eval_chunk(0xBEEF, 40, 0, members)
    got = ctx.read_losses(0, members)
    for at in (0, members // 2, members - 2):
        assert (got[at:at + 2] == O.eval_losses(ocfg, model, data, 40, 0xBEEF, at, 2)).all(), at
    ctx.close()
