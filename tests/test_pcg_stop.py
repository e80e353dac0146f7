"""The on-chip Jacobi-PCG stops at the iteration where the quotient of the
residuals passes the tolerance, also where that quotient underflows."""
import numpy as np
import pytest

from pic_b200 import deck
from pic_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


# tolerance squared, charge: an ordinary solve; a square that underflows to 0;
# a bound below the normal numbers; and one above them by little
@pytest.mark.parametrize("tol,charge", [(1e-10, 0.05), (1e-170, 1e100), (1e-140, 1e-20), (1e-146, 1.0), (1e-30, 1e-130)])
def test_stops_where_the_quotient_does(tol, charge, monkeypatch):
    n, h = 24, 0.01 / 16
    cfg = deck.config("tiny", ncx=n, ncy=n, Lx=n * h, Ly=n * h, objects=[], wall_V=(0.0,) * 4, pcg_tol=tol, pcg_maxit=20000)
    rng = np.random.default_rng(1)
    rho = charge * rng.standard_normal((n + 1) ** 2)
    got = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("PIC_PCG_SMEM", mode)
        sim = Simulation(cfg, load=False, capacity=[16, 16], mcc=False)
        try:
            phi = sim.mesh.array("phi_dirichlet").copy()
            sim.set_field("rho", rho)
            try:
                st = sim.ife_solve(phi)
                got[mode] = (st.iterations, st.ierr, st.rel_residual)
            except Exception as e:  # both have to fail alike
                got[mode] = str(e)
            got[mode + "phi"] = sim.field("phi")
        finally:
            sim.close()
    assert got["1"] == got["0"]
    assert np.array_equal(got["1phi"], got["0phi"])
