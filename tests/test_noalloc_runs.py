"""pic_deposit_noalloc against its fixed-point law in numpy, to the bit:
particles in runs of one element and in any order, counts around a thread's
four and a block's, arrays that are not 16-byte aligned, the walls."""
import numpy as np
import pytest

from pic_b200 import api

pytestmark = pytest.mark.gpu


def _law(nnx, nny, xmin, xmax, ymin, ymax, x, y, loc, vol, wq, L, n_ref):
    hx, hy = (xmax - xmin) / (nnx - 1), (ymax - ymin) / (nny - 1)
    rx, ry = (x - xmin) / hx, (y - ymin) / hy
    ok = (loc >= 0) & (rx >= 0) & (ry >= 0) & (rx < nnx) & (ry < nny)
    x, y, rx, ry = x[ok], y[ok], rx[ok], ry[ok]
    i, j = np.minimum(rx.astype(np.int64), nnx - 2), np.minimum(ry.astype(np.int64), nny - 2)
    x1, x2 = xmin + hx * i, xmin + hx * (i + 1)
    y1, y2 = ymin + hy * j, ymin + hy * (j + 1)
    dx, dy = (x - x1) / (x2 - x1), (y - y1) / (y2 - y1)
    xc, yc = 1.0 - dx, 1.0 - dy
    one = 2.0 ** 40
    q0, q1, q3 = (np.rint(w * one).astype(np.int64) for w in (xc * yc, dx * yc, xc * dy))
    acc = np.zeros(nnx * nny, np.int64)
    n1 = i * nny + j
    for n, q in ((n1, q0), (n1 + nny, q1), (n1 + nny + 1, (1 << 40) - (q0 + q1 + q3)), (n1 + 1, q3)):
        np.add.at(acc, n, q)
    return ((((wq * (acc * (1.0 / one))) / L) / L) / n_ref) / vol


@pytest.mark.parametrize("order", ["sorted", "unsorted", "mixed"])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 5, 127, 1024, 1027, 200003])
def test_deposit_matches_its_law(n, offset, order):
    import torch
    lib = api.load()
    nnx, nny, xmin, ymin = 23, 41, -1.7, 0.3
    xmax, ymax = xmin + 0.1 * (nnx - 1), ymin + 0.37 * (nny - 1)
    rng = np.random.default_rng(n + offset)
    cell = rng.integers(0, (nnx - 1) * (nny - 1), n)
    if order == "sorted":
        cell = np.sort(cell)
    elif order == "mixed":  # sorted with every third particle anywhere
        cell = np.where(np.arange(n) % 3 == 0, cell, np.sort(cell))
    x = xmin + 0.1 * (cell // (nny - 1) + rng.random(n))
    y = ymin + 0.37 * (cell % (nny - 1) + rng.random(n))
    x[::11], y[::13] = xmin, ymin
    x[1::17], y[1::19] = xmax, ymax
    if n > 4:
        x[4] = xmax + 0.5  # outside: not deposited
    loc = np.where(rng.random(n) < 0.1, -1, 0).astype(np.int32)
    vol = rng.random(nnx * nny) + 0.5

    def dev(a):
        t = torch.zeros(a.size + offset, dtype=torch.from_numpy(a).dtype, device="cuda")[offset:]
        t.copy_(torch.from_numpy(a))
        return t

    dx, dy, dl, dv = dev(x), dev(y), dev(loc), dev(vol)
    for use_loc in (True, False):
        out = torch.full((nnx * nny,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        api.check(lib.pic_deposit_noalloc(nnx, nny, xmin, xmax, ymin, ymax, n, dx.data_ptr(), dy.data_ptr(),
                                          dl.data_ptr() if use_loc else None, dv.data_ptr(), -0.013, 0.7, 1e15,
                                          out.data_ptr(), None), "pic_deposit_noalloc")
        torch.cuda.synchronize()
        want = _law(nnx, nny, xmin, xmax, ymin, ymax, x, y, loc if use_loc else np.zeros(n, np.int32), vol, -0.013,
                    0.7, 1e15)
        assert np.array_equal(out.cpu().numpy(), want)
