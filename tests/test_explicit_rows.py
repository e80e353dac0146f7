"""Explicit rows of the solver's operator: stored as stencils when the CSR
lists each row's 3x3 neighbours in column order, as column lists otherwise.
Both against the oracle, over walls whose nodes are unknowns (stencil
positions outside the grid) and r-z meshes (one stencil per radius)."""
import numpy as np
import pytest

import oracle_bind as ob
from pic_b200 import api, deck
from pic_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


def _swap_first_pair(mesh):
    """Swaps the first two entries of a full row: no longer in column order."""
    d = mesh.desc
    u = next(u for u in range(d.n_unknowns // 2, d.n_unknowns) if d.a_srow[u + 1] - d.a_srow[u] == 9)
    q = d.a_srow[u] - 1
    for a in (d.a_jcol, d.a_k):
        a[q], a[q + 1] = a[q + 1], a[q]


@pytest.mark.parametrize("persistent", ["1", "0"])
@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("name,ncx,ncy,walls", [("tiny", 16, 16, (1, 1, 1, 1)), ("tiny", 33, 17, (0, 0, 0, 1)),
                                                ("tiny", 17, 40, (1, 0, 0, 0)), ("tiny_axi", 16, 16, (1, 1, 0, 1)),
                                                ("tiny_axi", 37, 50, (0, 1, 0, 1))])
def test_solve_matches_oracle(name, ncx, ncy, walls, swap, persistent, monkeypatch):
    monkeypatch.setenv("PIC_PCG_PERSISTENT", persistent)
    h = 0.01 / 16
    obj = deck.ObjectSpec(api.PIC_SHAPE_CIRCLE, 0.5013 * ncx * h, 0.5471 * ncy * h, 0.2137 * min(ncx, ncy) * h, eps=4.0)
    cfg = deck.config(name, ncx=ncx, ncy=ncy, Lx=ncx * h, Ly=ncy * h, objects=[obj], wall_dirichlet=walls)

    class _Mesh(deck.Mesh):
        def __init__(self, cfg):
            super().__init__(cfg)
            if swap:
                _swap_first_pair(self)

    monkeypatch.setattr("pic_b200.simulation.Mesh", _Mesh)
    sim = Simulation(cfg, load=False, capacity=[16, 16], mcc=False)
    try:
        nn = sim.mesh.nn
        rho = 0.05 * np.random.default_rng(5).standard_normal(nn)
        phi0 = sim.mesh.array("phi_dirichlet").copy()
        sim.set_field("rho", rho)
        phi = phi0.copy()
        st = sim.ife_solve(phi)
        po, so = ob.pcg(sim.mesh.ptr, ob.rhs(sim.mesh.ptr, rho, nn), phi0, cfg.pcg_tol, cfg.pcg_maxit)
        assert st.ierr == 0 and st.iterations == so["iterations"]
        assert np.array_equal(phi, po)
    finally:
        sim.close()
