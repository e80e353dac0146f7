"""The mixed push takes one particle a thread where the bulk-staged form, two a
thread, would have a tile or less for each of its resident CTAs: the same bits
on both sides of that count, the MCC selection among them, and no slower than
the one-particle form asked for by name."""
import numpy as np
import pytest

from pic_b200 import api, deck
from pic_b200.simulation import Simulation

pytestmark = pytest.mark.gpu

FORMS = {"by count": {}, "bulk": {"PIC_PUSH_BULK": "1"}, "direct": {"PIC_PUSH_BULK": "0", "PIC_PUSH_STAGES": "0"}}


def _sim(name, n, form, monkeypatch, ncells=64):
    for k in ("PIC_PUSH_BULK", "PIC_PUSH_STAGES"):
        monkeypatch.delenv(k, raising=False)
    for k, v in FORMS[form].items():
        monkeypatch.setenv(k, v)
    L = 0.01 / 16 * ncells
    cfg = deck.config(name, ncx=ncells, ncy=ncells, Lx=L, Ly=L, objects=[], precision=api.PIC_PREC_MIXED, pcg_tol=1e-4,
                      ppc=max(1, n // ncells ** 2), sort_interval=1000, wall_particles=(0, 0, 0, 1))
    sim = Simulation(cfg, load=False, capacity=[n + 4096] * 2)
    rng = np.random.default_rng(n)
    m = sim.mesh
    for s in range(2):
        x, y = (0.001 + 0.998 * rng.random(n)) * m.hx * ncells, (0.001 + 0.998 * rng.random(n)) * m.hy * ncells
        v = rng.standard_normal((3, n)) * deck.species_params(cfg)[0][s][3]
        sim.upload(s, x, y, *[np.ascontiguousarray(c) for c in v])
        sim.sort(s)
    sim.initial_fields()
    return sim


@pytest.mark.parametrize("name", ["tiny", "tiny_axi"])
@pytest.mark.parametrize("n", [1, 255, 20011, 1184 * 256, 1184 * 256 + 1])
def test_same_bits_on_both_sides(name, n, monkeypatch):
    got = []
    for form in ("by count", "bulk"):
        sim = _sim(name, n, form, monkeypatch)
        try:
            out = []
            for _ in range(3):
                st = sim.step()
                out += [sim.field(f) for f in ("rho_e", "rho_i", "phi")]
                out += [[st.mcc.n_by_reaction[k][r] for k in range(2) for r in range(4)]]
            sim.move_all(0)
            for s in range(2):
                p = sim.download(s)
                out += [p[k] for k in ("x", "y", "vx", "vy", "vz", "loc", "id")] + [sim.count(s)]
            got.append(out)
        finally:
            sim.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_few_particles_take_no_longer_than_one_a_thread(monkeypatch):
    t = {}
    for form in ("by count", "direct"):
        sim = _sim("tiny", 20000, form, monkeypatch, ncells=128)
        try:
            for _ in range(5):
                sim.step()
            t[form] = min(sim.step().ms_push_kernel for _ in range(60))
        finally:
            sim.close()
    # the bulk form: 1.3 times
    assert t["by count"] <= 1.15 * t["direct"]
