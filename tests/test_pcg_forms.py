"""Jacobi-PCG's forms agree to the bit: the persistent kernel built for explicit
rows as stencils and as lists, against the two-kernel iteration."""
import numpy as np
import pytest

from pic_b200 import api, deck
from pic_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


def _solve(monkeypatch, name, ncx, ncy, env, swap=False, n_obj=1, tol=1e-4):
    for k in ("PIC_PCG_SMEM", "PIC_PCG_PERSISTENT"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    h = 0.01 / 16
    Lx, Ly = ncx * h, ncy * h
    k = int(np.ceil(np.sqrt(n_obj)))
    objs = [deck.ObjectSpec(api.PIC_SHAPE_CIRCLE, Lx * (a // k + 0.5013) / k, Ly * (a % k + 0.5471) / k,
                            0.3137 * min(Lx, Ly) / k, eps=1.5 + 0.37 * a) for a in range(n_obj)]
    cfg = deck.config(name, ncx=ncx, ncy=ncy, Lx=Lx, Ly=Ly, objects=objs, pcg_tol=tol)

    class _Mesh(deck.Mesh):
        def __init__(self, cfg):
            super().__init__(cfg)
            if swap:  # one row out of column order: explicit rows as lists
                d = self.desc
                u = next(u for u in range(d.n_unknowns // 2, d.n_unknowns) if d.a_srow[u + 1] - d.a_srow[u] == 9)
                q = d.a_srow[u] - 1
                for a in (d.a_jcol, d.a_k):
                    a[q], a[q + 1] = a[q + 1], a[q]

    monkeypatch.setattr("pic_b200.simulation.Mesh", _Mesh)
    sim = Simulation(cfg, load=False, capacity=[16, 16], mcc=False)
    try:
        phi = sim.mesh.array("phi_dirichlet").copy()
        sim.set_field("rho", 0.05 * np.random.default_rng(ncx).standard_normal((ncx + 1) * (ncy + 1)))
        st = sim.ife_solve(phi)
        return st.iterations, st.ierr, st.ms, phi
    finally:
        sim.close()


@pytest.mark.parametrize("name,ncx,ncy", [("tiny", 30, 33), ("tiny", 127, 8), ("tiny_axi", 40, 70), ("tiny", 210, 190)])
@pytest.mark.parametrize("swap", [False, True])
def test_persistent_matches_two_kernels(name, ncx, ncy, swap, monkeypatch):
    a = _solve(monkeypatch, name, ncx, ncy, {"PIC_PCG_SMEM": "0"}, swap)
    b = _solve(monkeypatch, name, ncx, ncy, {"PIC_PCG_PERSISTENT": "0"}, swap)
    assert a[:2] == b[:2] and a[1] == 0 and a[0] > 3
    assert np.array_equal(a[3], b[3])


# columns at the length where each number of chunks a CTA hands over to the
# chunked kernel (2 (nny + 1) halo values for 256, 512 and 1024 threads)
@pytest.mark.parametrize("ncx,ncy", [(12, 2557), (12, 2558), (40, 4605), (40, 4606), (70, 5629), (70, 5630)])
def test_long_columns_match_the_chunked_kernel(ncx, ncy, monkeypatch):
    a = _solve(monkeypatch, "tiny", ncx, ncy, {})
    b = _solve(monkeypatch, "tiny", ncx, ncy, {"PIC_PCG_SMEM": "0"})
    assert a[:2] == b[:2] and a[1] == 0 and a[0] > 3
    assert np.array_equal(a[3], b[3])


def test_long_columns_take_no_longer_than_in_the_chunked_kernel(monkeypatch):
    t = {}
    for mode in ("default", "0"):
        env = {} if mode == "default" else {"PIC_PCG_SMEM": "0"}
        t[mode] = min(_solve(monkeypatch, "tiny", 20, 6000, env)[2] for _ in range(4))
    # on chip 1.7 times
    assert t["default"] <= 1.25 * t["0"]
