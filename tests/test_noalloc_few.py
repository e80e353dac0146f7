"""The allocation-free deposit takes one particle a thread for few particles, or
few a node, and four for more: its fixed-point law to the bit on both sides of
the counts where it changes."""
import numpy as np
import pytest

from test_noalloc_runs import _law
from pic_b200 import api

pytestmark = pytest.mark.gpu

FEW = 148 * 2048


@pytest.mark.parametrize("nnx,nny,n", [(23, 41, FEW), (23, 41, FEW + 1), (500, 401, FEW + 1), (500, 401, 2 * 500 * 401 - 1),
                                       (500, 401, 2 * 500 * 401)])
@pytest.mark.parametrize("order", ["sorted", "unsorted"])
def test_both_sides_match_the_law(nnx, nny, n, order):
    import torch
    lib = api.load()
    rng = np.random.default_rng(n)
    cell = rng.integers(0, (nnx - 1) * (nny - 1), n)
    if order == "sorted":
        cell = np.sort(cell)
    xmax, ymax = 0.1 * (nnx - 1), 0.37 * (nny - 1)
    x, y = 0.1 * (cell // (nny - 1) + rng.random(n)), 0.37 * (cell % (nny - 1) + rng.random(n))
    loc = np.where(rng.random(n) < 0.05, -1, 0).astype(np.int32)
    vol = rng.random(nnx * nny) + 0.5
    t = [torch.from_numpy(a).cuda() for a in (x, y, loc, vol)]
    out = torch.full((nnx * nny,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    api.check(lib.pic_deposit_noalloc(nnx, nny, 0.0, xmax, 0.0, ymax, n, *[a.data_ptr() for a in t], -0.013, 0.7, 1e15,
                                      out.data_ptr(), None), "pic_deposit_noalloc")
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), _law(nnx, nny, 0.0, xmax, 0.0, ymax, x, y, loc, vol, -0.013, 0.7, 1e15))

