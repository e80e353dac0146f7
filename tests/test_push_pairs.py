"""The bulk-staged pushes take two particles a thread and deposit the pair
together: against one particle a thread, to the bit, for counts around a pair,
a warp's 64 and a tile's 256, in cell order and in any order, with absorbed
slots among them."""
import numpy as np
import pytest

from pic_b200 import api, deck
from pic_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,prec,env", [("tiny", api.PIC_PREC_FP64, "PIC_PUSH64_TILED"),
                                           ("tiny_axi", api.PIC_PREC_FP64, "PIC_PUSH64_TILED"),
                                           ("tiny", api.PIC_PREC_MIXED, "PIC_PUSH_BULK"),
                                           ("tiny_axi", api.PIC_PREC_MIXED, "PIC_PUSH_BULK")])
@pytest.mark.parametrize("order", ["sorted", "unsorted"])
@pytest.mark.parametrize("n", [1, 2, 3, 63, 65, 255, 257, 20011])
def test_pairs_match_single_particles(name, prec, env, order, n, monkeypatch):
    got = {}
    for mode in ("2" if env == "PIC_PUSH64_TILED" else "1", "0"):
        monkeypatch.setenv(env, mode)
        cfg = deck.config(name, precision=prec, pcg_tol=1e-3, sort_interval=1000)
        sim = Simulation(cfg, load=False, capacity=[n, n], mcc=False)
        try:
            rng = np.random.default_rng(n)
            m = sim.mesh
            for s in range(2):
                x, y = (0.001 + 0.998 * rng.random(n)) * m.hx * 16, (0.001 + 0.998 * rng.random(n)) * m.hy * 16
                v = rng.standard_normal((3, n)) * (1.0, 0.02)[s]
                sim.upload(s, x, y, *[np.ascontiguousarray(c) for c in v])
                if order == "sorted":
                    sim.sort(s)
            sim.initial_fields()
            out = []
            for _ in range(4):  # fast electrons leave: absorbed slots from the first step on
                sim.step()
                out += [sim.field(f) for f in ("rho_e", "rho_i", "phi")]
            sim.move_all(0)  # a push without a deposit
            for s in range(2):
                p = sim.download(s)
                out += [p[k] for k in ("x", "y", "vx", "vy", "vz", "loc", "id")] + [sim.count(s)]
            got[mode] = out
        finally:
            sim.close()
    a, b = got.values()
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
