"""Products that pairs of thread blocks form together (cta_group::2): the same losses as the two-kernel form, whose blocks work alone, for
every member, and as the CPU oracle for the members of the first and the last row tile.  The sizes: an odd number of row tiles (the last
pair forms one twice and stores it once), tiles of one member and of several, sub-tiles of 256 and of 128 columns, clusters of four
(a pair for each half of the columns), even and uneven halves."""
import numpy as np
import pytest

from common import load_oracle, load_pkg, make_case

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
