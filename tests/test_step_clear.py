"""A step clears all that its push adds to in one launch.  The densities it
leaves are those of a deposit that clears for itself, to the bit, for every
remainder of the node count by the 16-byte fill, with the energy accumulators
cleared only on the steps that deposit them, and the particle counts are those
of the slots that are still live."""
import numpy as np
import pytest

from pic_b200 import api, deck
from pic_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(16, 16), (17, 16), (17, 17), (16, 18)])
@pytest.mark.parametrize("diag_interval", [1, 3])
def test_step_clears_its_accumulators(cells, diag_interval):
    cfg = deck.config("tiny", ncx=cells[0], ncy=cells[1], pcg_tol=1e-3, sort_interval=1000,
                      diag_interval=diag_interval)
    n = 3001
    sim = Simulation(cfg, load=False, capacity=[n, n], mcc=False)
    try:
        rng = np.random.default_rng(cells[0] * 100 + cells[1])
        m = sim.mesh
        for s in range(2):
            x = (0.001 + 0.998 * rng.random(n)) * m.hx * cells[0]
            y = (0.001 + 0.998 * rng.random(n)) * m.hy * cells[1]
            v = rng.standard_normal((3, n)) * (1.0, 0.02)[s]
            sim.upload(s, x, y, *[np.ascontiguousarray(c) for c in v])
        sim.initial_fields()
        for _ in range(5):
            sim.step()
            rho, each = sim.field("rho"), [sim.field(f) for f in ("rho_e", "rho_i")]
            for s in range(2):
                p = sim.download(s)
                assert sim.count(s) == len(p["x"])
            sim.get_par_chg()
            assert np.array_equal(rho, sim.field("rho"))
            for f, u in zip(("rho_e", "rho_i"), each):
                assert np.array_equal(u, sim.field(f))
    finally:
        sim.close()
