"""Device pointers that are only as aligned as the interface asks for give the same bytes as aligned ones."""
import numpy as np
import pytest

from common import load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [4, 8, 12])
@pytest.mark.parametrize("n,rows_per_member,pairs", [(256, 32, 2), (384, 32, 3), (2048, 64, 40), (256, 48, 1)])
def test_projection_into_words(n, rows_per_member, pairs, offset):
    import torch
    pkg = load_pkg()
    ctx = pkg.Context(pkg.default_config(device_mask=15, population_size=64), 0, 2)
    rows, k = 2 * rows_per_member * pairs, 256
    g = torch.Generator(device="cuda")
    g.manual_seed(n + offset)
    x = torch.randint(-127, 128, (rows, k), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-127, 128, (k * n + offset,), generator=g, device="cuda", dtype=torch.int8)
    y = torch.empty(rows * n, dtype=torch.int8, device="cuda")
    z = torch.full((rows * n + 16,), 99, dtype=torch.int8, device="cuda")
    torch.cuda.synchronize()
    for out in (y.data_ptr(), z.data_ptr() + offset):
        ctx.perturbed_projection(x.data_ptr(), w.data_ptr() + offset, out, rows, k, n, rows_per_member, 5, 200, 201, 7, 9, on_device=True)
    z = z.cpu().numpy()
    assert (z[offset:offset + rows * n] == y.cpu().numpy()).all()
    assert (z[:offset] == 99).all() and (z[offset + rows * n:] == 99).all()
    ctx.close()


@pytest.mark.parametrize("offset", [1, 2, 3, 4])
@pytest.mark.parametrize("optimizer", [0, 1])
def test_matrix_update_of_weights_anywhere(optimizer, offset):
    import torch
    pkg = load_pkg()
    ctx = pkg.Context(pkg.default_config(device_mask=3, population_size=64), 0, 2)
    rows, cols, pairs = 128, 384, 100
    g = torch.Generator(device="cuda")
    g.manual_seed(offset)
    w = torch.randint(-127, 128, (rows * cols,), generator=g, device="cuda", dtype=torch.int8)
    v = torch.full((rows * cols + 8,), 99, dtype=torch.int8, device="cuda")
    v[offset:offset + rows * cols] = w
    opt = torch.randn(rows * cols, 3 - optimizer, generator=g, device="cuda")
    if not optimizer:
        opt[:, 1].square_()
    opt2 = opt.clone()
    fit = torch.randint(-1, 2, (pairs,), generator=g, device="cuda", dtype=torch.int32)
    torch.cuda.synchronize()
    n = [ctx.update_matrix(p, o.data_ptr(), rows, cols, 402, 403, 0, fit.data_ptr(), pairs, 7, 0.4, optimizer, False)
         for p, o in ((w.data_ptr(), opt), (v.data_ptr() + offset, opt2))]
    v = v.cpu().numpy()
    # the norm's terms are added in any order: a weight on a rounding boundary may differ under Muon
    assert (v[offset:offset + rows * cols] != w.cpu().numpy()).sum() <= (2 if optimizer else 0)
    assert abs(n[0] - n[1]) <= (2 if optimizer else 0) and n[0] > 0
    assert (v[:offset] == 99).all() and (v[offset + rows * cols:] == 99).all()
    ctx.close()
