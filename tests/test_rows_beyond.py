"""Row tables past what the other decks reach: more distinct stencils than
constant memory takes on a Cartesian mesh, more explicit rows a CTA of the
persistent flexible CG than its shared-memory table, and the FP32 form of the
column walk by its iterations."""
import numpy as np
import pytest

import oracle_bind as ob
from pic_b200 import api, deck
from pic_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


def _sim(monkeypatch, name, ncx, ncy, n_obj=1, lists=False, **over):
    h = 0.01 / 16
    Lx, Ly = ncx * h, ncy * h
    k = int(np.ceil(np.sqrt(n_obj)))
    objs = [deck.ObjectSpec(api.PIC_SHAPE_CIRCLE, Lx * (a // k + 0.5013) / k, Ly * (a % k + 0.5471) / k,
                            0.3137 * min(Lx, Ly) / k, eps=1.5 + 0.37 * a) for a in range(n_obj)]
    cfg = deck.config(name, ncx=ncx, ncy=ncy, Lx=Lx, Ly=Ly, objects=objs, **over)

    class _Mesh(deck.Mesh):
        def __init__(self, cfg):
            super().__init__(cfg)
            if lists:  # one row out of column order: explicit rows as lists
                d = self.desc
                u = next(u for u in range(d.n_unknowns // 2, d.n_unknowns) if d.a_srow[u + 1] - d.a_srow[u] == 9)
                q = d.a_srow[u] - 1
                for a in (d.a_jcol, d.a_k):
                    a[q], a[q + 1] = a[q + 1], a[q]

    monkeypatch.setattr("pic_b200.simulation.Mesh", _Mesh)
    return Simulation(cfg, load=False, capacity=[16, 16], mcc=False)


def _fcg(sim, **solver):
    try:
        sim.set_solver("fcg", window=1, omega=0.8, multigrid=True, **solver)
        sim.set_field("rho", 0.05 * np.random.default_rng(3).standard_normal(sim.mesh.nn))
        phi = sim.mesh.array("phi_dirichlet").copy()
        st = sim.ife_solve(phi)
        assert st.ierr == 0 and st.fallback == 0
        return st.iterations, phi
    finally:
        sim.close()


@pytest.mark.parametrize("smem", ["1", "0"])
@pytest.mark.parametrize("lists", [False, True])
def test_more_materials_than_constant_memory_match_oracle(lists, smem, monkeypatch):
    monkeypatch.setenv("PIC_PCG_SMEM", smem)
    sim = _sim(monkeypatch, "tiny", 100, 90, n_obj=25, lists=lists)
    try:
        rho = 0.05 * np.random.default_rng(5).standard_normal(sim.mesh.nn)
        phi0 = sim.mesh.array("phi_dirichlet").copy()
        sim.set_field("rho", rho)
        phi = phi0.copy()
        st = sim.ife_solve(phi)
        cfg = sim.cfg
        po, so = ob.pcg(sim.mesh.ptr, ob.rhs(sim.mesh.ptr, rho, sim.mesh.nn), phi0, cfg.pcg_tol, cfg.pcg_maxit)
        assert st.ierr == 0 and st.iterations == so["iterations"]
        assert np.array_equal(phi, po)
    finally:
        sim.close()


# 304 columns of 1217 radii: 1217 stencils, of which a CTA's table holds 1100
@pytest.mark.parametrize("name,ncx,ncy,n_obj", [("tiny_axi", 304, 1216, 1), ("tiny", 160, 192, 25)])
def test_fcg_matches_the_launched_kernels(name, ncx, ncy, n_obj, monkeypatch):
    got = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("PIC_FCG_PERSISTENT", mode)
        got[mode] = _fcg(_sim(monkeypatch, name, ncx, ncy, n_obj, pcg_tol=1e-10))
    # the bars of the multigrid tests: dot products in another order
    assert abs(got["1"][0] - got["0"][0]) <= 2
    assert np.abs(got["1"][1] - got["0"][1]).max() <= 1e-7 * np.abs(got["0"][1]).max()


def test_fp32_walk_converges_as_the_node_by_node_form(monkeypatch):
    got = {}
    for form in ("fp64", "walk", "lists"):
        prec = api.PIC_PREC_FP64 if form == "fp64" else api.PIC_PREC_MIXED
        sim = _sim(monkeypatch, "tiny", 128, 64, lists=form == "lists", precision=prec, pcg_tol=1e-10)
        got[form] = _fcg(sim, inner_fp32=form != "fp64")
    # the same FP32 arithmetic but for the order of sums: a few iterations in all;
    # restarts of the refinement and FP32 rounding together at most double the count
    assert abs(got["walk"][0] - got["lists"][0]) <= 3
    assert got["walk"][0] <= 2 * got["fp64"][0]
    for form in ("walk", "lists"):
        assert np.abs(got[form][1] - got["fp64"][1]).max() <= 1e-7 * np.abs(got["fp64"][1]).max()
