"""Quotients by known reciprocals (div_dev.h) where the reciprocal is out of its
range, a zero numerator among them: the division is taken."""
import numpy as np
import pytest

from test_noalloc_runs import _law
from pic_b200 import api, deck, simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [1e-45, 1e-41, 1e-39, 1e39, 1e41, 1e45])
def test_deposit_on_meshes_of_any_scale(h):
    import torch
    lib = api.load()
    nnx, nny = 9, 6
    xmax, ymax = h * (nnx - 1), 2.0 * h * (nny - 1)
    # every node, the lower walls (numerator 0) among them, and the cells' middles
    i, j = np.meshgrid(np.arange(nnx), np.arange(nny), indexing="ij")
    x = np.concatenate([xmax * (i.ravel() / (nnx - 1)), [0.0, 0.5 * h, 0.0]])
    y = np.concatenate([ymax * (j.ravel() / (nny - 1)), [0.0, 0.0, h]])
    t = [torch.from_numpy(a).cuda() for a in (x, y, np.ones(nnx * nny))]
    out = torch.zeros(nnx * nny, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    api.check(lib.pic_deposit_noalloc(nnx, nny, 0.0, xmax, 0.0, ymax, x.size, t[0].data_ptr(), t[1].data_ptr(), None,
                                      t[2].data_ptr(), 1.0, 1.0, 1.0, out.data_ptr(), None), "pic_deposit_noalloc")
    torch.cuda.synchronize()
    want = np.ones((nnx, nny))
    want[0, 0] += 1.0                       # (0, 0)
    want[:2, 0] += 0.5                      # (h/2, 0)
    want[0, :2] += 0.5                      # (0, h): the cells are 2h tall
    # positions are within an ulp or two of the nodes, charges within 2^-40
    assert np.abs(out.cpu().numpy().reshape(nnx, nny) - want).max() < 1e-11


@pytest.mark.parametrize("quarters,steps", [(3, 0), (4, -1), (13, -1), (27, 0)])
def test_deposit_in_cells_a_unit_short_of_a_power_of_two(quarters, steps):
    """xmin off zero by a few quarters of 2^-53: the first cell's width rounds
    to 1 - 2^-53, the divisor whose reciprocal Newton's steps leave a place low."""
    import torch
    lib = api.load()
    nnx, nny = 3, 4
    xmin = 0.0625 + quarters * 2.0 ** -55
    xmax = xmin + 2.0
    for _ in range(-steps):
        xmax = np.nextafter(xmax, 0.0)
    assert (xmin + (xmax - xmin) / 2) - xmin == 1.0 - 2.0 ** -53
    # a power of two into the cell; (1 - dy) dx 2^40 on one side of k + 1/2, by
    # the last place of dx
    k = np.arange(0, 64, 2)
    y = 1.0 - (2.0 * k + 1.0) * 2.0 ** -37
    x = np.full(y.size, xmin + 0.0625)
    assert np.all(x - xmin == 0.0625)
    n, vol, loc = x.size, np.ones(nnx * nny), np.zeros(x.size, np.int32)
    t = [torch.from_numpy(a).cuda() for a in (x, y, vol)]
    out = torch.zeros(nnx * nny, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    api.check(lib.pic_deposit_noalloc(nnx, nny, xmin, xmax, 0.0, nny - 1.0, n, t[0].data_ptr(), t[1].data_ptr(), None,
                                      t[2].data_ptr(), 1.0, 1.0, 1.0, out.data_ptr(), None), "pic_deposit_noalloc")
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), _law(nnx, nny, xmin, xmax, 0.0, nny - 1.0, x, y, loc, vol, 1.0, 1.0, 1.0))


@pytest.mark.parametrize("scale", [2.0 ** -150, 2.0 ** -136, 2.0 ** 140])
def test_onchip_pcg_with_a_tiny_or_huge_diagonal(scale, monkeypatch):
    class Scaled(deck.Mesh):
        def __init__(self, cfg):
            super().__init__(cfg)
            d = self.desc
            for ptr, n in ((d.a_k, d.nnz), (d.a_diag, d.n_unknowns)):
                a = np.ctypeslib.as_array(ptr, shape=(n,))  # in place
                a *= scale

    monkeypatch.setattr(simulation, "Mesh", Scaled)
    n, h = 48, 0.01 / 16
    cfg = deck.config("tiny", ncx=n, ncy=n, Lx=n * h, Ly=n * h, objects=[], wall_V=(0.0,) * 4, pcg_tol=1e-6, pcg_maxit=500)
    rho = np.zeros((n + 1, n + 1))
    rho[3:6, 3:6] = 0.05  # elsewhere the residual is 0 until the iterations reach it
    got = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("PIC_PCG_SMEM", mode)
        sim = simulation.Simulation(cfg, load=False, capacity=[16, 16], mcc=False)
        try:
            phi = sim.mesh.array("phi_dirichlet").copy()
            sim.set_field("rho", rho.reshape(-1))
            st = sim.ife_solve(phi)
            got[mode] = (st.iterations, st.ierr, phi)
        finally:
            sim.close()
    assert got["1"][:2] == got["0"][:2]
    assert np.array_equal(got["1"][2], got["0"][2], equal_nan=True)
    assert np.isfinite(got["0"][2]).all() and np.any(got["0"][2])
