"""Newton-Schulz of one matrix update against the same steps in float64 on the float32 starting point (votes of zero fitness
vanish, so the momentum is known): the smallest tile, several tiles of the triangle, contractions of one and of many stages,
square, wide and tall.  Bound: each of the ten products is within 2^-23 of the exact one relative to its operands (six
partial products of 2^-24 weight, chains of four truncating additions, rounded sums above), errors enter additively and
a step's derivative stays below one on average: 10 * 2^-23."""
import numpy as np
import pytest

from common import load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(128, 128), (128, 384), (640, 256), (384, 384), (256, 1024), (1024, 512)])
def test_newton_schulz_against_float64(rows, cols):
    import torch
    pkg = load_pkg()
    ctx = pkg.Context(pkg.default_config(device_mask=3, population_size=64, adam_weight_decay=0.0), 0, 2)
    g = torch.Generator(device="cuda")
    g.manual_seed(rows + cols)
    m0 = torch.randn(rows, cols, generator=g, device="cuda")
    opt = torch.zeros(rows * cols, 2, device="cuda")
    opt[:, 0] = m0.reshape(rows // 4, 4, cols).permute(0, 2, 1).reshape(-1)         # packed order [rows/4][cols][4]
    w = torch.zeros(rows * cols, dtype=torch.int8, device="cuda")
    fit = torch.zeros(32, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    # rate 1 and no decay: the accumulator ends as minus the update (entries are far below one, nothing is quantised away)
    n = ctx.update_matrix(w.data_ptr(), opt.data_ptr(), rows, cols, 402, 403, 0, fit.data_ptr(), 32, 7, 1.0, 1, False)
    un = lambda v: v.reshape(rows // 4, cols, 4).permute(0, 2, 1).reshape(rows, cols)      # noqa: E731
    m, u = un(opt[:, 0]), -un(opt[:, 1]).double()
    assert n == 0 and (w == 0).all()
    x = (m / m.double().square().sum().sqrt().float()).double()
    for _ in range(5):
        if rows < cols:
            x = 0.5 * (3 * x - x @ x.T @ x)
        else:
            x = 0.5 * (3 * x - x @ (x.T @ x))
    err = float((u - x).norm() / x.norm())
    assert err < 10 * 2.0 ** -23, err
    ctx.close()


@pytest.mark.parametrize("rows,cols", [(128, 128), (256, 384), (128, 2048), (4096, 128)])
def test_newton_schulz_is_closer_than_a_chain_of_multiply_adds(rows, cols):
    """The error of the six-term products against the same steps in float64, beside that of float32 products that feed one
    accumulator in the order of the contraction (measured: 3.8e-7 to 4.5e-7 against 4.6e-7 to 6.4e-7)."""
    import torch

    def chain(a, b):
        acc = torch.zeros(a.shape[0], b.shape[1], device="cuda")
        for t in range(a.shape[1]):
            acc = torch.addcmul(acc, a[:, t:t + 1], b[t:t + 1, :])
        return acc

    def steps(x, product):
        k = min(x.shape)
        for _ in range(5):
            g = 3 * torch.eye(k, dtype=x.dtype, device="cuda") - (product(x, x.T) if rows < cols else product(x.T, x))
            x = 0.5 * (product(g, x) if rows < cols else product(x, g))
        return x

    pkg = load_pkg()
    ctx = pkg.Context(pkg.default_config(device_mask=3, population_size=64, adam_weight_decay=0.0), 0, 2)
    g = torch.Generator(device="cuda")
    g.manual_seed(rows + cols)
    opt = torch.zeros(rows * cols, 2, device="cuda")
    opt[:, 0] = torch.randn(rows * cols, generator=g, device="cuda")
    w = torch.zeros(rows * cols, dtype=torch.int8, device="cuda")
    fit = torch.zeros(32, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.update_matrix(w.data_ptr(), opt.data_ptr(), rows, cols, 402, 403, 0, fit.data_ptr(), 32, 7, 1.0, 1, False)
    m, u = (v.reshape(rows // 4, cols, 4).permute(0, 2, 1).reshape(rows, cols) for v in (opt[:, 0], -opt[:, 1]))
    x0 = m / m.double().square().sum().sqrt().float()
    x = steps(x0.double(), torch.matmul)
    ours, chained = float((u - x).norm() / x.norm()), float((steps(x0, chain) - x).norm() / x.norm())
    assert ours <= chained, (ours, chained)
    ctx.close()
