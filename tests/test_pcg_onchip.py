"""The on-chip Jacobi-PCG (every CTA's chunks in registers and shared memory)
against the one-chunk-at-a-time persistent kernel, which the oracle pins: the
same chunk partials and sums, so the same iterations and the same bits."""
import numpy as np
import pytest

from pic_b200 import api, deck
from pic_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


def _solves(cfg, rho):
    sim = Simulation(cfg, load=False, capacity=[16, 16], mcc=False)
    try:
        out = []
        phi = sim.mesh.array("phi_dirichlet").copy()
        for r in rho:  # the second solve follows the tags of the first
            sim.set_field("rho", r)
            st = sim.ife_solve(phi)
            out.append((st.iterations, st.ierr, st.rel_residual, phi.copy()))
        return out
    finally:
        sim.close()


# chunks (1024 nodes) a CTA owns: one CTA, a ragged last chunk, one, two,
# three or four and five to eight of them; strips wider than a CTA's nodes
# (columns of 1501 nodes); r-z, where almost every row is an explicit one
@pytest.mark.parametrize("name,ncx,ncy", [("tiny", 16, 16), ("tiny", 31, 31), ("tiny", 32, 32), ("tiny", 67, 45),
                                          ("tiny_axi", 75, 50), ("tiny", 30, 1500), ("tiny", 1500, 30),
                                          ("tiny", 390, 400), ("tiny_axi", 300, 201), ("tiny", 700, 630),
                                          ("tiny", 900, 880)])
def test_onchip_pcg_matches_the_chunked_kernel(name, ncx, ncy, monkeypatch):
    h = 0.01 / 16
    R = min(ncx, ncy) * h
    obj = deck.ObjectSpec(api.PIC_SHAPE_CIRCLE, 0.5013 * ncx * h, 0.5471 * ncy * h, 0.2137 * R, eps=4.0)
    cfg = deck.config(name, ncx=ncx, ncy=ncy, Lx=ncx * h, Ly=ncy * h, objects=[obj], pcg_tol=1e-4)
    rng = np.random.default_rng(ncx)
    rho = 0.05 * rng.standard_normal((2, (ncx + 1) * (ncy + 1)))
    got = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("PIC_PCG_SMEM", mode)
        got[mode] = _solves(cfg, rho)
    for a, b in zip(got["1"], got["0"]):
        assert a[:3] == b[:3] and a[1] == 0 and a[0] > 3
        assert np.array_equal(a[3], b[3])
