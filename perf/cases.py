"""What the framework is measured on: the work its users have it do, through its
public entry points, over the range of sizes they run.

Kinds of case
  run      a short run from its initial particles on a small deck: upload,
           initial fields, ten steps, download
  steps    one sort period of the main loop (Simulation.step) of a running
           simulation, and the fields it leaves read back
  loop     the caller's own main loop over the reference's subroutines
           (MoveAll, GetParChg_2D, IFE_Solve_2D, GetEField_SIDG_PPR, MCC, sort)
  solve    IFE_Solve_2D from host Rho and Phi, Phi read back
  diag     the output routines: column profiles, spectra, velocity moments
  deposit  the allocation-free charge deposit on device pointers
  train    one optimiser step of the learned preconditioner's network
  precond  one application of the whole learned preconditioner

The library holds one simulation per process.  Several inputs are held at once
here, so every state that needs a simulation has a copy of the library of its
own (loaded from memory), taken from a pool and given back with the state.
"""
from __future__ import annotations

import ctypes as C
import math
import os
from contextlib import contextmanager

import numpy as np
import torch

from pic_b200 import api, deck, unet
from pic_b200.simulation import Simulation

# --------------------------------------------------------------------------
# the cases


def listed():
    return [
        # the smallest deck a user starts with (64^2, one dielectric disk, the
        # reference's Jacobi-PCG at 1e-10): a short restart, where launches,
        # copies and waits count more than bandwidth
        {"name": "run_64", "kind": "run", "deck": "cfg1", "ncx": 64, "ncy": 64, "ppc": 50, "precision": "fp64",
         "solver": "jpcg", "tol": 1e-10},
        # a short axisymmetric run at an odd size, FP64
        {"name": "run_rz_75x50", "kind": "run", "deck": "torus", "ncx": 75, "ncy": 50, "ppc": 33,
         "precision": "fp64", "solver": "jpcg", "tol": 1e-10},
        # a Fortran-style caller that owns the loop, a grid that is no power of
        # two, absorbing and reflecting walls, MCC
        {"name": "loop_200x136", "kind": "loop", "deck": "box", "ncx": 200, "ncy": 136, "ppc": 30,
         "precision": "fp64", "solver": "jpcg", "tol": 1e-10},
        # the 512^2 deck with a conductor on the plain path: the step is
        # Jacobi-PCG for nine tenths of its time
        {"name": "steps_512_jpcg", "kind": "steps", "deck": "cfg2", "ncx": 512, "ncy": 512, "ppc": 24,
         "precision": "fp64", "solver": "jpcg", "tol": 1e-10, "period": 10},
        # an ordinary mixed-precision run: the disk deck at 512^2
        {"name": "steps_512_mixed", "kind": "steps", "deck": "cfg3", "ncx": 512, "ncy": 512, "ppc": 32,
         "precision": "mixed", "solver": "mg", "tol": 1e-8, "period": 10},
        # the headline: 1024^2, eight ellipses, 101.7M particles, FP64
        {"name": "steps_1024_fp64", "kind": "steps", "deck": "cfg4", "ncx": 1024, "ncy": 1024, "ppc": 64,
         "precision": "fp64", "solver": "mg", "tol": 1e-8, "period": 20},
        # the driven axisymmetric cell, mixed precision
        {"name": "steps_rz_mixed", "kind": "steps", "deck": "cfg5", "ncx": 2048, "ncy": 1024, "ppc": 16,
         "precision": "mixed", "solver": "mg", "tol": 1e-8, "period": 10},
        # the Poisson solve alone, called with host arrays as the reference calls it
        {"name": "solve_1024_mg", "kind": "solve", "deck": "cfg4", "ncx": 1024, "ncy": 1024, "ppc": 0,
         "precision": "fp64", "solver": "mg", "tol": 1e-8},
        # the output step of a running simulation
        {"name": "diag_256", "kind": "diag", "deck": "cfg1", "ncx": 256, "ncy": 256, "ppc": 100, "precision": "fp64",
         "solver": "jpcg", "tol": 1e-10, "nbins": 100, "ncols": 1024},
        # a caller with particles of its own in device memory
        {"name": "deposit_257x200", "kind": "deposit", "nnx": 257, "nny": 200, "n": 3000001, "order": "sorted"},
        # one optimiser step on the default training batch
        {"name": "train_4x128", "kind": "train", "batch": 4, "crop": 128},
        # the learned preconditioner on the headline grid
        {"name": "precond_1024", "kind": "precond", "deck": "cfg4", "ncx": 1024, "ncy": 1024, "ppc": 0,
         "precision": "fp64", "solver": "mg", "tol": 1e-8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "steps", "steps", "steps", "loop", "solve", "diag", "deposit", "deposit", "train", "precond"])
    if kind == "deposit":
        return {"kind": kind, "nnx": _log(rng, 17, 700), "nny": _log(rng, 17, 700), "n": _log(rng, 1e3, 2e7),
                "order": rng.choice(["sorted", "unsorted"])}
    if kind == "train":
        return {"kind": kind, "batch": rng.randint(1, 8), "crop": rng.randint(32, 160)}
    c = {"kind": kind}
    # grids: any size for Jacobi-PCG, sizes that halve for the multigrid
    mg = kind == "precond" or (kind in ("steps", "solve") and rng.random() < 0.7)
    if mg:
        k = 2 ** rng.randint(1, 4)
        c.update(deck=rng.choice(["disks", "torus"]) if kind != "precond" else "disks",
                 ncx=k * rng.randint(12, 64), ncy=k * rng.randint(12, 64))
    elif kind in ("run", "loop"):
        c.update(deck="box" if kind == "loop" else rng.choice(["disks", "torus"]), ncx=_log(rng, 16, 150), ncy=_log(rng, 16, 150))
    else:
        c.update(deck=rng.choice(["disks", "torus"]), ncx=_log(rng, 48, 512), ncy=_log(rng, 48, 512))
    most = {"run": 5e5, "loop": 2e6, "steps": 1.2e7, "diag": 1.2e7}.get(kind, 0.0)
    c["ppc"] = max(1, min(_log(rng, 4, 100), int(most / (c["ncx"] * c["ncy"])))) if most else 0
    c["precision"] = rng.choice(["fp64", "mixed"])
    c["solver"], c["tol"] = ("mg", 1e-8) if mg else ("jpcg", 1e-10)
    if kind == "steps":
        c["period"] = rng.choice([5, 10, 20])
    if kind == "diag":
        c["precision"] = "fp64"
        c["nbins"], c["ncols"] = rng.choice([50, 100, 1000]), rng.choice([64, 500, 1024])
    return c


# --------------------------------------------------------------------------
# decks


def _config(case) -> deck.Config:
    name, over = case["deck"], dict(ncx=case["ncx"], ncy=case["ncy"], pcg_tol=case["tol"], pcg_maxit=50000,
                                    ppc=max(case["ppc"], 1), sort_interval=case.get("period", 10),
                                    precision=api.PIC_PREC_MIXED if case["precision"] == "mixed" else api.PIC_PREC_FP64)
    if name.startswith("cfg"):
        return deck.config(name, **over)
    hx = 0.01 / 16  # the cell of the small test decks
    Lx, Ly = hx * case["ncx"], hx * case["ncy"]
    R = min(Lx, Ly)
    over.update(Lx=Lx, Ly=Ly, n0=1e15, Te_eV=2.0, seed=3)
    if case["kind"] in ("steps", "loop"):  # the sides absorb, bottom (not the r-z axis) and top reflect
        over.update(wall_particles=(0, 0, 0, 1) if name == "torus" else (0, 0, 1, 1))
    # centres and radii off the lattice: the interface must miss the vertices
    if name == "disks":
        return deck.config("tiny", objects=[
            deck.ObjectSpec(api.PIC_SHAPE_CIRCLE, 0.3013 * Lx, 0.5171 * Ly, 0.1337 * R, eps=4.0),
            deck.ObjectSpec(api.PIC_SHAPE_CIRCLE, 0.7059 * Lx, 0.4583 * Ly, 0.1513 * R, eps=2.0)], **over)
    if name == "torus":
        return deck.config("tiny_axi", objects=[
            deck.ObjectSpec(api.PIC_SHAPE_CIRCLE, 0.5013 * Lx, 0.5471 * Ly, 0.2137 * R, eps=4.0)], **over)
    if name == "box":  # no object
        return deck.config("tiny", objects=[], **over)
    raise KeyError(name)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _particles(cfg, mesh, species, seed):
    """A quiet Maxwellian plasma outside the objects, cell by cell (uniform in
    volume on an r-z mesh), drawn on the device: x, y, vx, vy, vz."""
    g = _generator(seed * 7919 + species)
    f64 = dict(dtype=torch.float64, device="cuda")
    sigma = deck.species_params(cfg)[0][species][3]
    cells = torch.arange(cfg.ncx * cfg.ncy, device="cuda")
    if cfg.delta == 1:  # a ring's share of the cylinder
        mean = cfg.ppc * (2.0 * (cells % cfg.ncy) + 1.0) / cfg.ncy
        cells = cells.repeat_interleave(torch.floor(mean + torch.rand(cells.numel(), generator=g, **f64)).long())
    else:
        cells = cells.repeat_interleave(cfg.ppc)
    n = cells.numel()
    x = ((cells // cfg.ncy) + torch.rand(n, generator=g, **f64)) * mesh.hx
    j = (cells % cfg.ncy).to(torch.float64)
    if cfg.delta == 1:
        r0, r1 = j * mesh.hy, (j + 1.0) * mesh.hy
        y = torch.sqrt(r0 * r0 + torch.rand(n, generator=g, **f64) * (r1 * r1 - r0 * r0))
    else:
        y = (j + torch.rand(n, generator=g, **f64)) * mesh.hy
    keep = torch.ones(n, dtype=torch.bool, device="cuda")
    for k in range(mesh.deck.n_objects):
        o = mesh.deck.objects[k]
        if o.shape == api.PIC_SHAPE_BOX:
            keep &= ~((x > o.cx) & (x < o.a) & (y > o.cy) & (y < o.b))
        else:
            c, s = math.cos(o.angle), math.sin(o.angle)
            u, v = (x - o.cx) * c + (y - o.cy) * s, -(x - o.cx) * s + (y - o.cy) * c
            keep &= ~(u * u / (o.a * o.a) + v * v / (o.b * o.b) < 1.0)
    x, y = x[keep], y[keep]
    v = [torch.randn(x.numel(), generator=g, **f64) * sigma for _ in range(3)]
    return [x, y] + v


# --------------------------------------------------------------------------
# simulations, each on a copy of the library of its own

_pool, _in_memory = [], []


def _library():
    if _pool:
        return _pool.pop()
    if not _in_memory:
        _in_memory.append(None)
        return api.load()
    fd = os.memfd_create("libpicgpu")  # kept open: its number names the copy
    with open(api.LIB_PATH, "rb") as f:
        data = memoryview(f.read())
    while data:
        data = data[os.write(fd, data):]
    _in_memory.append(fd)
    mine = api._lib, api.LIB_PATH
    api._lib, api.LIB_PATH = None, "/proc/self/fd/%d" % fd
    try:
        return api.load()
    finally:
        api._lib, api.LIB_PATH = mine


@contextmanager
def _using(lib):
    mine, api._lib = api._lib, lib
    try:
        yield
    finally:
        api._lib = mine


class _State:
    """A simulation and what a case needs beside it."""

    def __init__(self, case, seed):
        self.case, self.lib, self.sim = case, _library(), None
        try:
            with _using(self.lib):
                self._build(seed)
        except BaseException:
            self.close()
            raise

    def _build(self, seed):
        case = self.case
        self.cfg = cfg = _config(case)
        n = 2 if case["ppc"] else 0
        cap = [1024, 1024]
        if n:
            most = cfg.ncx * cfg.ncy * (cfg.ppc + (1 if cfg.delta == 1 else 0))
            cap = [int(most * 1.1) + 65536] * 2  # room for ionisation
        self.sim = sim = Simulation(cfg, load=False, capacity=cap, mcc=None if n else False)
        self.host = []
        st = C.c_void_p()
        api.check(self.lib.pic_cuda_stream(C.byref(st)), "pic_cuda_stream")
        self.stream = torch.cuda.ExternalStream(st.value)
        for s in range(n):
            p = _particles(cfg, sim.mesh, s, seed)
            host = [t.cpu().numpy() for t in p]
            sim.upload(s, *host)
            if case["kind"] == "run":
                self.host.append(host)
            del p
        torch.cuda.empty_cache()
        if case["kind"] == "run":
            self.own = [[np.zeros(c) for _ in range(5)] + [np.zeros(c, np.int32), np.zeros(c, np.uint32)] for c in cap]
        elif n and case["precision"] == "fp64":
            self.own = [[torch.zeros(c, dtype=t, device="cuda") for t in [torch.float64] * 5 + [torch.int32] * 2] for c in cap]
        if case["solver"] == "mg":
            sim.set_solver("fcg", window=1, multigrid=True, omega=0.8)
        if n and case["kind"] != "run":
            for s in range(n):
                sim.sort(s)
            sim.initial_fields()
        nn = sim.mesh.nn
        self.fields = [torch.zeros(nn, dtype=torch.float64).pin_memory().numpy() for _ in range(4)]
        if case["kind"] == "solve":
            self._solve_inputs(seed)
        if case["kind"] == "precond":
            self.lp = unet.LearnedPreconditioner(sim, seed=seed, window=4, multigrid=True, omega=0.8)
            self.r = _charge(sim.mesh, seed).reshape(-1).cuda() * self.lp.mask_f
            self.z = torch.zeros_like(self.r)
        torch.cuda.synchronize()

    def _solve_inputs(self, seed):
        mesh = self.sim.mesh
        self.rho = _charge(mesh, seed).reshape(-1).pin_memory().numpy()
        self.guess = torch.from_numpy(mesh.array("phi_dirichlet")).pin_memory().numpy()
        self.phi = torch.zeros(mesh.nn, dtype=torch.float64).pin_memory().numpy()

    def particles(self):
        """The particle arrays (FP64 layout), copied on the device from where
        they are into the caller's own, zero past the last particle."""
        for s in range(2):
            ptr, n = (C.c_void_p * 7)(), C.c_int64()
            api.check(self.lib.pic_particle_device_ptrs(s, ptr, C.byref(n)), "pic_particle_device_ptrs")
            with torch.cuda.stream(self.stream):  # between this step's kernels and the next one's
                for k, t in enumerate(self.own[s]):
                    view = torch.as_tensor(unet.DeviceArray(ptr[k], n.value, "<f8" if k < 5 else "<i4"), device="cuda")
                    t[:n.value].copy_(view)
                    t[n.value:].zero_()
        return self.own

    def download(self):
        """The particles in host arrays of the caller's, zero past the last."""
        for s in range(2):
            n = C.c_int64()
            a = self.own[s]
            api.check(self.lib.pic_download_particles(s, a[0].size, *[api.dptr(v) for v in a[:5]], api.iptr(a[5]),
                                                      api.uptr(a[6]), C.byref(n)), "pic_download_particles")
        return [[v if v.dtype != np.uint32 else v.view(np.int32) for v in a] for a in self.own]

    def close(self):
        lib, self.lib = self.lib, None
        if lib is None:
            return
        if self.sim is not None:
            torch.cuda.synchronize()
            self.lp = None  # its graphs run on the simulation's stream
            with _using(lib):
                self.sim.close()
        _pool.append(lib)

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def _charge(mesh, seed):
    """A smooth charge with the grain of a finite number of particles."""
    rng = np.random.default_rng(seed)
    x = np.linspace(0.0, 1.0, mesh.nnx)[:, None]
    y = np.linspace(0.0, 1.0, mesh.nny)[None, :]
    rho = 0.05 * rng.standard_normal((mesh.nnx, mesh.nny))
    for _ in range(6):
        a, b = rng.integers(1, 6, 2)
        rho += 0.1 * rng.standard_normal() * np.sin(math.pi * a * x) * np.sin(math.pi * b * y)
    return torch.from_numpy(np.ascontiguousarray(rho))


class _Deposit:
    def __init__(self, case, seed):
        g = _generator(seed)
        f64 = dict(dtype=torch.float64, device="cuda")
        self.nnx, self.nny, n = case["nnx"], case["nny"], case["n"]
        self.hx, self.hy = 0.37, 0.41
        self.xmax, self.ymax = self.hx * (self.nnx - 1), self.hy * (self.nny - 1)
        ex, ey = self.nnx - 1, self.nny - 1
        cell = torch.randint(0, ex * ey, (n,), generator=g, device="cuda")
        if case["order"] == "sorted":
            cell = cell.sort().values
        self.x = (((cell // ey) + torch.rand(n, generator=g, **f64)) * self.hx).clamp(max=self.xmax)
        self.y = (((cell % ey) + torch.rand(n, generator=g, **f64)) * self.hy).clamp(max=self.ymax)
        # a few slots are free (absorbed particles)
        self.loc = torch.where(torch.rand(n, generator=g, **f64) < 0.02, -1, cell).to(torch.int32)
        wx, wy = torch.full((self.nnx,), self.hx, **f64), torch.full((self.nny,), self.hy, **f64)
        wx[[0, -1]] *= 0.5
        wy[[0, -1]] *= 0.5
        self.vol = (wx[:, None] * wy[None, :]).reshape(-1).contiguous()
        self.rho = torch.zeros_like(self.vol)
        self.weight = -1.0 / max(n / (ex * ey), 1e-3)


class _Train:
    def __init__(self, case, seed):
        b, c = case["batch"], case["crop"]
        g = _generator(seed)
        self.net = unet.UNet(seed=seed, stream=None)
        self.net._ensure(b, c, c)
        r = torch.randn(b, c, c, dtype=torch.float64, device="cuda", generator=g)
        self.target = torch.randn(b, c, c, dtype=torch.float64, device="cuda", generator=g).cumsum(1).contiguous()
        static = torch.randn(b, c, c, 3, device="cuda", generator=g).contiguous()
        self.mask = (torch.rand(b, c, c, device="cuda", generator=g) > 0.02).to(torch.int32)
        scratch = torch.zeros(unet.UNET_RMS_SCRATCH, dtype=torch.float64, device="cuda")
        sc = torch.zeros(b, 2, dtype=torch.float64, device="cuda")
        self.scale = torch.zeros(b, 2, dtype=torch.float64, device="cuda")
        self.loss = torch.zeros(2, dtype=torch.float64, device="cuda")
        L, p = self.net.lib, unet._p
        for k in range(b):
            unet._ck(L.unet_rms(c * c, p(r[k]), p(self.mask[k]), p(scratch), p(sc[k]), None), "rms")
            unet._ck(L.unet_rms(c * c, p(self.target[k]), p(self.mask[k]), p(scratch), p(self.scale[k]), None), "rms")
            unet._ck(L.unet_features(c, c, p(r[k]), p(sc[k]), p(static[k]), p(self.net.a["x0"][k]), None), "features")


def prepare(case, seed):
    if case["kind"] == "deposit":
        return case, _Deposit(case, seed)
    if case["kind"] == "train":
        return case, _Train(case, seed)
    return case, _State(case, seed)


# --------------------------------------------------------------------------
# one pass


def run(state):
    case, s = state
    kind = case["kind"]
    if kind == "deposit":
        api.check(api.load().pic_deposit_noalloc(s.nnx, s.nny, 0.0, s.xmax, 0.0, s.ymax, s.x.numel(), s.x.data_ptr(),
                                                 s.y.data_ptr(), s.loc.data_ptr(), s.vol.data_ptr(), s.weight, 1.0, 1.0,
                                                 s.rho.data_ptr(), None), "pic_deposit_noalloc")
        return s.rho
    if kind == "train":
        return _train(s)
    with _using(s.lib):
        return {"run": _run, "steps": _steps, "loop": _loop, "solve": _solve, "diag": _diag, "precond": _precond}[kind](s)


def _run(s):
    sim = s.sim
    for k in range(2):
        sim.upload(k, *s.host[k])
    sim.set_field("phi", np.zeros(sim.mesh.nn))
    sim.step_index = 0
    sim.initial_fields()
    for _ in range(10):
        st = sim.step()
    return {"phi": sim.field("phi"), "rho": sim.field("rho"), "n": [int(st.n_particles[k]) for k in range(2)],
            "particles": s.download()}


def _steps(s):
    for _ in range(s.cfg.sort_interval):
        st = s.sim.step()
    rho, phi, efx, efy = s.fields
    api.check(s.lib.pic_get_fields_async(api.dptr(rho), api.dptr(phi), api.dptr(efx), api.dptr(efy)), "pic_get_fields_async")
    api.check(s.lib.pic_wait_fields(), "pic_wait_fields")
    out = {"rho": rho, "phi": phi, "efx": efx, "efy": efy, "n": [int(st.n_particles[k]) for k in range(2)],
           "collisions": [int(st.mcc.n_by_reaction[k][r]) for k in range(2) for r in range(4)]}
    if s.case["precision"] == "fp64":
        out["particles"] = s.particles()
    return out


def _loop(s):
    sim = s.sim
    rho, phi, efx, efy = s.fields
    for _ in range(5):
        for k in range(2):
            sim.move_all(k)
        sim.get_par_chg(rho)
        sim.ife_solve(phi)
        sim.get_efield_ppr(efx, efy)
        sim.step_index += 1
        sim.mcc(sim.step_index)
    for k in range(2):
        sim.sort(k)
    out = {"rho": rho, "phi": phi, "efx": efx, "efy": efy, "n": [sim.count(k) for k in range(2)]}
    if s.case["precision"] == "fp64":
        out["particles"] = s.particles()
    return out


def _solve(s):
    api.check(s.lib.pic_set_field_async(0, api.dptr(s.rho)), "pic_set_field_async")
    api.check(s.lib.pic_set_field_async(1, api.dptr(s.guess)), "pic_set_field_async")
    s.sim.ife_solve()
    api.check(s.lib.pic_get_fields_async(None, api.dptr(s.phi), None, None), "pic_get_fields_async")
    api.check(s.lib.pic_wait_fields(), "pic_wait_fields")
    return s.phi


def _diag(s):
    sim, c = s.sim, s.case
    out = {"average_x": sim.average_x()}
    for k in range(2):
        out["spectrum%d" % k] = sim.energy_spectrum(k, c["nbins"], 10.0, (10.0, 0.1)[k])
        out["moments%d" % k] = sim.velocity_moments(k, c["ncols"])
    return out


def _train(s):
    net, p = s.net, unet._p
    b, c = s.target.shape[0], s.target.shape[1]
    net.zero_grad()
    s.loss.zero_()
    net.forward()
    for k in range(b):
        part = slice(k * c * c, (k + 1) * c * c)
        unet._ck(net.lib.unet_loss(c * c, p(net.z[part]), p(s.target[k]), p(s.scale[k]), p(s.mask[k]), p(net.gz[part]),
                                   p(s.loss), None), "loss")
    net.backward()
    net.adam(1e-3)
    return {"z": net.z, "loss": s.loss, "grad": {k: v["g"] for k, v in net.params.items()},
            "weights": {k: v["p"] for k, v in net.params.items()}}


def _precond(s):
    with torch.cuda.stream(s.lp.tstream):
        api.check(s.lib.pic_precond_apply(1, unet._p(s.r), unet._p(s.z)), "pic_precond_apply")
    return s.z


# --------------------------------------------------------------------------
# what a pass cannot do without


def _free_share(cfg):
    if cfg.delta == 1:
        return 1.0
    round_ = [o for o in cfg.objects if o.shape != api.PIC_SHAPE_BOX]
    return 1.0 - float(sum(math.pi * o.a * (o.b or o.a) for o in round_)) / (cfg.Lx * cfg.Ly)


def work(case):
    kind = case["kind"]
    if kind == "deposit":
        nn = case["nnx"] * case["nny"]
        return {"bytes": 20 * case["n"] + 16 * nn, "flops": 30 * case["n"]}
    if kind == "train":
        px = case["batch"] * case["crop"] ** 2
        level = {"e0": 1, "e1": 4, "b": 16, "d1": 4, "d0": 1}
        mac = sum(9 * ci * co / level[nm[:-1]] for nm, ci, co in unet.LAYERS)
        act = 2 * sum((ci + co) / level[nm[:-1]] for nm, ci, co in unet.LAYERS)
        return {"bytes": 3 * act * px, "flops": 3 * 2 * mac * px}
    cfg = _config(case)
    nn = (cfg.ncx + 1) * (cfg.ncy + 1)
    n = 2 * cfg.ncx * cfg.ncy * case["ppc"] * _free_share(cfg)
    fp64 = case["precision"] == "fp64"
    # a push reads and writes position, velocity and cell; a sort moves a particle whole
    push = (88 if cfg.delta == 1 else 72) if fp64 else (48 if cfg.delta == 1 else 40)
    moved = 96 if fp64 else 56
    # per step and node: charge out, potential in and out, fields and recovery coefficients out
    node = 8 * (2 + 1 + 2 + 2 + 5)
    if kind == "run":
        return {"bytes": 10 * (n * push + nn * node) + n * (2 * 48 + moved), "flops": 10 * (150 * n + 200 * nn)}
    if kind in ("steps", "loop"):
        k = cfg.sort_interval if kind == "steps" else 5
        return {"bytes": k * (n * push + nn * node) + n * moved, "flops": k * (150 * n + 200 * nn)}
    if kind == "solve":
        return {"bytes": 24 * nn, "flops": 200 * nn}
    if kind == "diag":
        return {"bytes": n * 40 + nn * 64, "flops": 40 * n}
    level = {"e0": 1, "e1": 4, "b": 16, "d1": 4, "d0": 1}
    mac = sum(9 * ci * co / level[nm[:-1]] for nm, ci, co in unet.LAYERS)
    act = 2 * sum((ci + co) / level[nm[:-1]] for nm, ci, co in unet.LAYERS)
    return {"bytes": (16 + act) * nn, "flops": (2 * mac + 200) * nn}


# --------------------------------------------------------------------------
# the same in 64 bits, in plain torch and numpy


def exact(case, seed):
    kind = case["kind"]
    if kind == "deposit":
        return _exact_deposit(_Deposit(case, seed))
    if kind == "train":
        return _exact_train(_Train(case, seed))
    if kind == "solve":
        return _exact_solve(case, seed)
    if kind == "diag":
        return _exact_diag(case, seed)
    # a run of the whole step, or the V-cycle with its 16-bit coarse inverse
    # around a 16-bit network: no plain 64-bit counterpart
    return None


def _exact_deposit(s):
    live = s.loc >= 0
    x, y = s.x[live] / s.hx, s.y[live] / s.hy
    i = x.floor().clamp(max=s.nnx - 2)
    j = y.floor().clamp(max=s.nny - 2)
    a, b = x - i, y - j
    n = (i * s.nny + j).long()
    q = torch.zeros_like(s.vol)
    for d, w in ((0, (1 - a) * (1 - b)), (s.nny, a * (1 - b)), (s.nny + 1, a * b), (1, (1 - a) * b)):
        q.index_add_(0, n + d, w)
    return s.weight * q / s.vol


def _exact_train(s):
    F = torch.nn.functional
    P = {}
    for k, v in s.net.params.items():
        P[k] = (v["p"] if k.startswith("head") else v["bf"]).double().clone().requires_grad_(True)

    def conv(name, x):
        return torch.relu(F.conv2d(x, P[name + ".w"].permute(0, 3, 1, 2), P[name + ".b"], padding=1))

    def pool(x):
        h, w = x.shape[2:]
        ones = torch.ones(1, 1, h, w, dtype=x.dtype, device=x.device)
        pad = (0, w % 2, 0, h % 2)
        return F.avg_pool2d(F.pad(x, pad), 2) / F.avg_pool2d(F.pad(ones, pad), 2)

    def up(lo, skip):
        u = lo.repeat_interleave(2, 2).repeat_interleave(2, 3)[:, :, :skip.shape[2], :skip.shape[3]]
        return torch.cat([u, skip], 1)

    x = s.net.a["x0"].double().permute(0, 3, 1, 2)
    e0 = conv("e0b", conv("e0a", x))
    e1 = conv("e1b", conv("e1a", pool(e0)))
    d = conv("bb", conv("ba", pool(e1)))
    d = conv("d1b", conv("d1a", up(d, e1)))
    d = conv("d0b", conv("d0a", up(d, e0)))
    z = (d * P["head.w"][None, :, None, None]).sum(1) + P["head.b"]
    m = (s.mask > 0).double()
    t = s.target / s.scale[:, 0].view(-1, 1, 1)
    loss = (m * (z - t) ** 2).sum()
    loss.backward()
    grad = {k: v.grad for k, v in P.items()}
    # the first Adam step
    weights = {k: v["p"].double() - 1e-3 * grad[k] / (grad[k].abs() + 1e-8) for k, v in s.net.params.items()}
    for k in weights:
        if k.endswith(".b"):  # from zero: one step is the sign of the gradient
            weights[k] = None
    return {"z": z.detach().reshape(-1), "loss": torch.stack([loss.detach(), (m * t * t).sum()]), "grad": grad, "weights": weights}


def _exact_solve(case, seed):
    """A phi = M rho - fixed - A_xt phi_D by conjugate gradients to rounding."""
    with _using(api.load()):
        mesh = deck.Mesh(_config(case))
        nnx, nny = mesh.nnx, mesh.nny
        dev = dict(device="cuda")
        A = {k: torch.from_numpy(mesh.array(k)).to(**dev) for k in
             ("node_type", "element_index", "phi_dirichlet", "a_srow", "a_jcol", "a_k", "xt_srow", "xt_jcol", "xt_k", "rhs_fix", "mass_q1",
              "ife_mass", "mass_rows") if k != "mass_rows" or mesh.desc.delta == 1}
        rho = _charge(mesh, seed).reshape(-1).cuda()
        mesh.close()
    ne = (nnx - 1) * (nny - 1)
    e = torch.arange(ne, **dev)
    n1 = (e // (nny - 1)) * nny + e % (nny - 1)
    corner = torch.stack([n1, n1 + nny, n1 + nny + 1, n1 + 1], 1)
    M = A["mass_rows"].view(-1, 4, 4)[e % (nny - 1)] if "mass_rows" in A else A["mass_q1"].view(1, 4, 4).expand(ne, 4, 4)
    M = M.clone()
    cut = A["element_index"] > 0
    M[cut] = A["ife_mass"].view(-1, 4, 4)[A["element_index"][cut].long() - 1]
    load = torch.zeros(nnx * nny, dtype=torch.float64, **dev)
    load.index_add_(0, corner.reshape(-1), torch.einsum("ejk,ek->ej", M, rho[corner]).reshape(-1))
    free = A["node_type"] > 0
    unknown = A["node_type"][free].long() - 1
    nu = A["a_srow"].numel() - 1

    def csr(rows, cols, vals, n):
        return torch.sparse_csr_tensor(rows.long() - 1, cols.long() - 1, vals, size=(nu, n))

    b = torch.zeros(nu, dtype=torch.float64, **dev)
    b[unknown] = load[free]
    K = csr(A["a_srow"], A["a_jcol"], A["a_k"], nu)
    b = b - A["rhs_fix"] - csr(A["xt_srow"], A["xt_jcol"], A["xt_k"], nnx * nny) @ A["phi_dirichlet"]
    rows = torch.repeat_interleave(torch.arange(nu, **dev), (A["a_srow"][1:] - A["a_srow"][:-1]).long())
    diag = torch.zeros(nu, dtype=torch.float64, **dev)
    on = rows == A["a_jcol"].long() - 1
    diag[rows[on]] = A["a_k"][on]
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rz = torch.dot(r, z)
    stop = 1e-13 * b.norm()
    for k in range(20000):
        q = K @ p
        a = rz / torch.dot(p, q)
        x += a * p
        r -= a * q
        if k % 100 == 99 and bool(r.norm() <= stop):
            break
        z = r / diag
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    phi = A["phi_dirichlet"].clone()
    phi[free] = x[unknown]
    return phi.cpu().numpy()


def _exact_diag(case, seed):
    cfg = _config(case)
    with _using(api.load()):
        mesh = deck.Mesh(cfg)
        p = [_particles(cfg, mesh, k, seed) for k in range(2)]
        mesh.close()
    out = {"average_x": None}
    for k in range(2):
        x, v = p[k][0], torch.stack(p[k][2:5])
        b = x.floor().clamp(0, case["ncols"] - 1).long()
        n = torch.bincount(b, minlength=case["ncols"])
        d = torch.maximum(n, torch.ones_like(n))
        drift = torch.stack([torch.bincount(b, weights=w, minlength=case["ncols"]) for w in v]) / d
        dv = v - drift[:, b]
        thermal = torch.sqrt(torch.stack([torch.bincount(b, weights=w * w, minlength=case["ncols"]) for w in dv]) / d)
        out["spectrum%d" % k] = None
        out["moments%d" % k] = [n, drift, thermal]
    return out
