"""A bulk-staged push refills a stage of its tile ring by bulk copies (the async
proxy) after the threads' ordinary accesses to it.  Where those are stores too,
every thread has to fence its own before the barrier that closes the tile.
Read from the source, and on the GPU with every stage refilled several times:
bit for bit against one particle a thread."""
import os
import re

import numpy as np
import pytest

from pic_b200 import api, deck
from pic_b200.simulation import Simulation

SRC = os.path.join(os.path.dirname(api.__file__), "csrc", "picgpu.cu")
FENCE = 'asm volatile("fence.proxy.async.shared::cta;\\n" ::: "memory");'


@pytest.mark.parametrize("kernel", ["k_push_bulk", "k_push_mixed_bulk"])
def test_stores_to_the_tile_are_fenced_by_every_thread(kernel):
    text = open(SRC).read()
    start = text.index("{", text.index(") " + kernel + "("))
    end = text.index("push_select_flush(s, sel_buf);\n}", start)
    body = re.sub(r"//[^\n]*", "", text[start:end])
    loop = body[body.index("for (int64_t t = blockIdx.x; t < ntiles"):]
    if not re.search(r"\bC\.\w+\[[^\]]*\] = ", loop):
        return  # the tile is only read
    barrier = loop.rindex("__syncthreads();")
    fence = loop.rindex(FENCE)
    # straight before the barrier, at the loop's own level, past the last use of the tile
    assert loop[fence + len(FENCE):barrier].strip() == ""
    assert loop[:fence].count("{") - loop[:fence].count("}") == 1
    assert not re.search(r"\bC\.", loop[fence:])


@pytest.mark.gpu
@pytest.mark.parametrize("name,prec,env", [("tiny", api.PIC_PREC_FP64, "PIC_PUSH64_TILED"),
                                           ("tiny_axi", api.PIC_PREC_FP64, "PIC_PUSH64_TILED"),
                                           ("tiny", api.PIC_PREC_MIXED, "PIC_PUSH_BULK"),
                                           ("tiny_axi", api.PIC_PREC_MIXED, "PIC_PUSH_BULK")])
def test_refilled_stages_match_single_particles(name, prec, env, monkeypatch):
    n = 2_500_001  # 9,766 tiles: several for each resident CTA, the last one of one particle
    got = {}
    for mode in ("2" if env == "PIC_PUSH64_TILED" else "1", "0"):
        monkeypatch.setenv(env, mode)
        cfg = deck.config(name, precision=prec, pcg_tol=1e-3, sort_interval=1000)
        sim = Simulation(cfg, load=False, capacity=[n, 1], mcc=False)
        try:
            rng = np.random.default_rng(7)
            m = sim.mesh
            x, y = (0.001 + 0.998 * rng.random(n)) * m.hx * 16, (0.001 + 0.998 * rng.random(n)) * m.hy * 16
            v = rng.standard_normal((3, n))
            sim.upload(0, x, y, *[np.ascontiguousarray(c) for c in v])
            sim.sort(0)
            sim.initial_fields()
            out = []
            for _ in range(3):
                sim.step()
                out.append(sim.field("rho_e"))
            p = sim.download(0)
            got[mode] = out + [p[k] for k in ("x", "y", "vx", "vy", "loc", "id")]
        finally:
            sim.close()
    a, b = got.values()
    for u, w in zip(a, b):
        assert np.array_equal(u, w)
