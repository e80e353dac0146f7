"""The persistent flexible CG, whose fine-grid phases walk columns in blocks of
rows, against its launch-per-operation path: row counts around a block and the
rest done node by node, few columns, walls of unknowns, r-z (every row explicit),
explicit rows kept as lists, the two-level space, FP32 inner iterations.  The
two paths sum dot products in other orders: the same iterations within 2 and
potentials within 1e-7, the bars of the multigrid tests."""
import numpy as np
import pytest

from pic_b200 import api, deck
from pic_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


def _solve(cfg, rho, swap, **solver):
    sim = Simulation(cfg, load=False, capacity=[16, 16], mcc=False)
    try:
        if solver.pop("inner", False):
            solver["inner_fp32"] = True
        sim.set_solver("fcg", window=1, omega=0.8, **solver)
        sim.set_field("rho", rho)
        phi = sim.mesh.array("phi_dirichlet").copy()
        st = sim.ife_solve(phi)
        assert st.ierr == 0 and st.fallback == 0
        return st.iterations, phi
    finally:
        sim.close()


@pytest.mark.parametrize("name,ncx,ncy,walls,kind", [
    ("tiny", 48, 32, (1, 1, 1, 1), "mg"), ("tiny", 96, 64, (1, 1, 1, 1), "mg"), ("tiny", 32, 512, (1, 1, 1, 1), "mg"),
    ("tiny", 32, 576, (0, 0, 0, 1), "mg"), ("tiny", 32, 1024, (1, 0, 0, 0), "mg"), ("tiny", 512, 32, (1, 1, 1, 1), "mg"),
    ("tiny_axi", 96, 128, (1, 1, 0, 1), "mg"), ("tiny_axi", 32, 544, (0, 1, 0, 1), "mg"),
    ("tiny", 128, 192, (1, 1, 0, 1), "list"), ("tiny", 128, 128, (1, 1, 1, 1), "coarse"),
    ("tiny", 128, 64, (1, 1, 1, 1), "fp32")])
def test_column_walk_matches_the_launched_kernels(name, ncx, ncy, walls, kind, monkeypatch):
    h = 0.01 / 16
    R = min(ncx, ncy) * h
    obj = deck.ObjectSpec(api.PIC_SHAPE_CIRCLE, 0.5013 * ncx * h, 0.5471 * ncy * h, 0.2137 * R, eps=4.0)
    cfg = deck.config(name, ncx=ncx, ncy=ncy, Lx=ncx * h, Ly=ncy * h, objects=[obj], wall_dirichlet=walls,
                      pcg_tol=1e-10, precision=api.PIC_PREC_MIXED if kind == "fp32" else api.PIC_PREC_FP64)

    class _Mesh(deck.Mesh):
        def __init__(self, cfg):
            super().__init__(cfg)
            if kind == "list":  # one row out of column order: explicit rows as lists
                d = self.desc
                u = next(u for u in range(d.n_unknowns // 2, d.n_unknowns) if d.a_srow[u + 1] - d.a_srow[u] == 9)
                q = d.a_srow[u] - 1
                for a in (d.a_jcol, d.a_k):
                    a[q], a[q + 1] = a[q + 1], a[q]

    monkeypatch.setattr("pic_b200.simulation.Mesh", _Mesh)
    rho = 0.05 * np.random.default_rng(ncx + ncy).standard_normal((ncx + 1) * (ncy + 1))
    solver = {"coarse_cells": 16} if kind == "coarse" else {"multigrid": True, "max_coarse_nodes": 1200}
    if kind == "fp32":
        solver["inner"] = True
    got = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("PIC_FCG_PERSISTENT", mode)
        got[mode] = _solve(cfg, rho, kind == "list", **dict(solver))
    # FP32 iterations run in the persistent kernel only
    slack = 10_000 if kind == "fp32" else 2
    assert abs(got["1"][0] - got["0"][0]) <= slack
    assert np.abs(got["1"][1] - got["0"][1]).max() <= 1e-7 * np.abs(got["0"][1]).max()
