"""The work that programs have this package do, as timed cases.

A case is a dict of plain values; ``prepare`` loads what a program holds before
its time loop, ``run`` is one pass of that loop through the public classes
(``CudaSim``, ``CudaBatch``, ``CudaSim1D``, ``AdjointSim``), and ``exact`` is the
same pass in 64 bits, in plain torch.  A state goes on from pass to pass, as a
simulation does.

Kinds:

- ``em2d``      the 2-D step, periodic: thermal and two-stream plasmas
- ``wakefield`` the 2-D step under a moving window, a Gaussian laser in a cold
                plasma that enters at the right edge
- ``scan``      independent two-stream runs of different sizes stepped together
- ``report``    the densities a diagnostic dump takes from a species
- ``em1d``      the 1-D step on the wakefield deck
- ``adjoint``   the gradient of the final field energy
"""
import math

import numpy as np
import torch

from zpic_gb300 import adjoint, batch, em1d_gpu
from zpic_gb300._zc import PART_DTYPE, CudaBatch, CudaSim

F64 = torch.float64


def listed():
    return [
        # the smallest run of the parity decks (two streams, 32 x 24 cells, 4 particles a cell and species, both
        # filters), one step a call as an interactive session steps it: launches and waits are all there is
        dict(name="deck32x24_step", kind="em2d", nx=32, ny=24, ppcx=2, ppcy=2, nspec=2, uth=0.1, drift=0.6, dt=0.07,
             filter="compensated", level=2, fast=False, tile="16x16", det=False, graphs=False, ext=0.0, steps=1,
             energy=False),
        # the Weibel deck (128^2, two streams of 16 particles a cell): a program that looks at the energies every step
        dict(name="weibel128_step_energy", kind="em2d", nx=128, ny=128, ppcx=4, ppcy=4, nspec=2, uth=0.1, drift=0.6,
             dt=0.07, filter="none", level=0, fast=False, tile="16x16", det=False, graphs=False, ext=0.0, steps=1,
             energy=True),
        # the same deck in blocks of replayed steps, as a long run of a small grid goes
        dict(name="weibel128_blocks", kind="em2d", nx=128, ny=128, ppcx=4, ppcy=4, nspec=2, uth=0.1, drift=0.6,
             dt=0.07, filter="none", level=0, fast=False, tile="16x16", det=False, graphs=True, ext=0.0, steps=32,
             energy=True),
        # the throughput workload: 2048^2 thermal plasma, 67 M particles, compensated filter, fast build
        dict(name="thermal2048_blocks", kind="em2d", nx=2048, ny=2048, ppcx=4, ppcy=4, nspec=1, uth=0.05, drift=0.0,
             dt=0.05, filter="compensated", level=1, fast=True, tile="32x16", det=False, graphs=True, ext=0.0,
             steps=16, energy=False),
        # sizes that divide by nothing, defaults of the class, 9 particles a cell, a magnetised plasma
        dict(name="magnetised1021x517", kind="em2d", nx=1021, ny=517, ppcx=3, ppcy=3, nspec=1, uth=0.1, drift=0.0,
             dt=0.06, filter="binomial", level=1, fast=False, tile="16x16", det=False, graphs=False, ext=0.5, steps=5,
             energy=True),
        # bit-reproducible deposition
        dict(name="deterministic512", kind="em2d", nx=512, ny=512, ppcx=4, ppcy=4, nspec=1, uth=0.05, drift=0.0,
             dt=0.05, filter="compensated", level=1, fast=True, tile="32x16", det=True, graphs=True, ext=0.0, steps=16,
             energy=False),
        # laser wakefield, 2000 x 256 cells, moving window with the column drawn on the device; the plasma already
        # under the pulse, as it is for all but the first steps of such a run
        dict(name="wakefield2000x256", kind="wakefield", nx=2000, ny=256, ppcx=4, ppcy=2, start=10.0, level=4,
             fast=True, tile="32x16", graphs=True, steps=16),
        # a parameter scan: two-stream runs of 64 to 256 cells an axis and 4 to 64 particles a cell, stepped together
        dict(name="scan24", kind="scan", runs=24, steps=12, sort_every=6, tile="32x16", table=2024),
        # charge and phase space of a species, as a report writes them
        dict(name="report512", kind="report", nx=512, ny=512, ppcx=4, ppcy=4, uth=0.05, pha_nx=512, pha_nu=128),
        # the 1-D wakefield deck: 1000 cells, 128 particles a cell, blocks of replayed steps
        dict(name="em1d_wakefield", kind="em1d", nx=1000, ppc=128, start=10.0, level=4, steps=32),
        # gradient of the field energy with respect to every particle, checkpointed
        dict(name="adjoint256", kind="adjoint", nx=256, ny=256, ppcx=4, ppcy=4, uth=0.05, steps=40, every=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["em2d", "em2d", "em2d", "wakefield", "scan", "report", "em1d", "adjoint"])
    tile = rng.choice(["16x16", "32x16"])
    if kind == "em2d":
        while True:
            nx, ny = _log(rng, 24, 2048), _log(rng, 24, 2048)
            ppcx, ppcy, nspec = rng.randint(1, 8), rng.randint(1, 8), rng.choice([1, 1, 2])
            if nx * ny * ppcx * ppcy * nspec <= 30_000_000:
                break
        filt = rng.choice(["none", "binomial", "compensated"])
        return dict(kind=kind, nx=nx, ny=ny, ppcx=ppcx, ppcy=ppcy, nspec=nspec, uth=round(rng.uniform(0.02, 0.2), 3),
                    drift=round(rng.uniform(0.2, 0.8), 2) if nspec == 2 else 0.0, dt=round(rng.uniform(0.04, 0.068), 3),
                    filter=filt, level=0 if filt == "none" else rng.randint(1, 4), fast=rng.random() < 0.5, tile=tile,
                    det=rng.random() < 0.15, graphs=rng.random() < 0.5, ext=rng.choice([0.0, 0.0, 0.0, 0.3]),
                    steps=rng.choice([1, 4, 7, 16]), energy=rng.random() < 0.5)
    if kind == "wakefield":
        nx = rng.randint(1400, 2400)
        return dict(kind=kind, nx=nx, ny=_log(rng, 48, 300), ppcx=rng.randint(2, 4), ppcy=rng.randint(1, 3),
                    start=round(nx * WAKE["dx"] * rng.uniform(0.1, 0.35), 2), level=rng.randint(1, 4),
                    fast=rng.random() < 0.5, tile=tile, graphs=rng.random() < 0.5, steps=rng.choice([4, 16]))
    if kind == "scan":
        return dict(kind=kind, runs=rng.randint(4, 28), steps=rng.choice([8, 12, 16]), sort_every=rng.choice([4, 6, 8]),
                    tile=tile, table=rng.randint(1, 10_000))
    if kind == "report":
        return dict(kind=kind, nx=_log(rng, 64, 800), ny=_log(rng, 64, 800), ppcx=rng.randint(1, 6),
                    ppcy=rng.randint(1, 6), uth=round(rng.uniform(0.02, 0.2), 3), pha_nx=rng.randint(32, 1024),
                    pha_nu=rng.randint(16, 300))
    if kind == "em1d":
        return dict(kind=kind, nx=rng.randint(900, 2400), ppc=rng.randint(8, 160), start=round(rng.uniform(4.0, 16.0), 2),
                    level=rng.randint(1, 4), steps=rng.choice([8, 16, 32, 50]))
    return dict(kind=kind, nx=_log(rng, 32, 256), ny=_log(rng, 32, 256), ppcx=rng.randint(1, 4), ppcy=rng.randint(1, 4),
                uth=round(rng.uniform(0.02, 0.1), 3), steps=rng.randint(5, 30), every=rng.choice([5, 10, 20]))


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _f(v):
    """the float32 value a handle keeps of v"""
    return float(np.float32(v))


def _gen(seed, k=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + k)


def _tile(c):
    return tuple(int(v) for v in c["tile"].split("x"))


def _plasma(nx, ny, ppcx, ppcy, uth, drift, gen, i0=0.0):
    """cells, in-cell positions and momenta of a species: the loading lattice
    of every cell right of column i0, thermal momenta with each cell's mean
    taken off, a drift along z (float32 values, particle by particle)"""
    npc, ncell = ppcx * ppcy, nx * ny
    cell = torch.arange(ncell, device="cuda", dtype=torch.int32)
    lx = ((torch.arange(ppcx, device="cuda") + 0.5) / ppcx).float().repeat(ppcy)
    ly = ((torch.arange(ppcy, device="cuda") + 0.5) / ppcy).float().repeat_interleave(ppcx)
    ix, iy = (cell % nx).repeat_interleave(npc), (cell // nx).repeat_interleave(npc)
    x, y = lx.repeat(ncell), ly.repeat(ncell)
    if uth > 0:
        u = uth * torch.randn((3, ncell, npc), generator=gen, device="cuda")
        if npc > 1:
            u -= u.mean(-1, keepdim=True)
        u = u.reshape(3, -1)
    else:
        u = torch.zeros((3, ncell * npc), device="cuda")
    u[2] += drift
    p = dict(ix=ix, iy=iy, x=x, y=y, ux=u[0], uy=u[1], uz=u[2])
    if i0 > 0:
        keep = ix + x > np.float32(i0)
        p = {k: v[keep] for k, v in p.items()}
    return p


def _records(p):
    """the particles as host records"""
    cols = [p[k].contiguous().view(torch.int32) for k in ("ix", "iy", "x", "y", "ux", "uy", "uz")]
    return torch.stack(cols, dim=1).cpu().numpy().reshape(-1).view(PART_DTYPE)


def _species(c, seed):
    """[(charge of a particle, particles)] of a periodic case"""
    nspec = c.get("nspec", 1)
    q = -1.0 / (c["ppcx"] * c["ppcy"])
    return [(q, _plasma(c["nx"], c["ny"], c["ppcx"], c["ppcy"], c["uth"], (1 - 2 * k) * c.get("drift", 0.0),
                        _gen(seed, k))) for k in range(nspec)]


def _laser(c, seed):
    """the wakefield decks' pulse, its strength and polarisation from the seed"""
    g = _gen(seed, 77)
    r = torch.rand(2, generator=g, device="cuda").cpu()
    return dict(start=17.0, fwhm=2.0, a0=1.5 + float(r[0]), omega0=10.0, polarization=math.pi * float(r[1]))


WAKE = dict(dx=0.02, dy=0.2, dt=0.014)
PULSE = dict(W0=4.0, focus=20.0)


def _window(c):
    nx, ny = c["nx"], c["ny"]
    box = (nx * WAKE["dx"], ny * WAKE["dy"])
    shift = (nx - 2000) * WAKE["dx"]  # the pulse keeps its distance from the right edge
    return box, shift


def _scan_table(c):
    return batch.weibel_scan(n_runs=c["runs"], steps=c["steps"], seed=c["table"])


# ---------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------
class _Device:
    """device memory of a simulation, for torch: a tensor made from it keeps
    this object, and so the simulation that owns the memory"""

    def __init__(self, sim, ptr, shape, strides):
        self.sim = sim
        self.__cuda_array_interface__ = dict(data=(int(ptr), False), shape=shape, typestr="<f4",
                                             strides=tuple(4 * s for s in strides), version=3)


class _Grids:
    """the interior of a simulation's E, B and J, in place on the device"""

    def __init__(self, sim):
        self.sim, self.seen = sim, {}

    def _view(self, v, ptr, planes):
        key = (ptr, planes)
        if key not in self.seen:
            nx, ny = self.sim.nx
            at = ptr + 4 * (v.pitch + 1)
            mem = _Device(self.sim, at, (planes, ny, nx), (v.plane, v.pitch, 1))
            self.seen[key] = torch.as_tensor(mem, device="cuda")
        return self.seen[key]

    def fields(self):
        v = self.sim.grid_view()
        return self._view(v, v.E, 6)  # Ex Ey Ez Bx By Bz

    def all(self):
        v = self.sim.grid_view()
        return {"EB": self._view(v, v.E, 6), "J": self._view(v, v.J, 3)}


def _sim2d(c, seed):
    nx, ny = c["nx"], c["ny"]
    sim = CudaSim((nx, ny), (nx * 0.1, ny * 0.1), c.get("dt", 0.05), tile=_tile(c) if "tile" in c else (16, 16),
                  fast_math=c.get("fast", False), deterministic=c.get("det", False))
    for q, p in _species(c, seed):
        sim.add_species(-1.0, q, (c["ppcx"], c["ppcy"]), _records(p))
    return sim


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind in ("em2d", "report"):
        sim = _sim2d(c, seed)
        if c.get("filter", "none") != "none":
            sim.set_smooth(c["filter"], c["level"], c["filter"], c["level"])
        if c.get("ext", 0.0):
            sim.set_ext_fld(B_type="uniform", B_0=(0.0, 0.0, c["ext"]))
        if c.get("graphs"):
            sim.set_graphs(True)
        return dict(c=c, sim=sim, grids=_Grids(sim))
    if kind == "wakefield":
        nx, ny = c["nx"], c["ny"]
        box, shift = _window(c)
        sim = CudaSim((nx, ny), box, WAKE["dt"], tile=_tile(c), fast_math=c["fast"])
        q = -1.0 / (c["ppcx"] * c["ppcy"])
        p = _plasma(nx, ny, c["ppcx"], c["ppcy"], 0.0, 0.0, None, i0=_f(c["start"]) / _f(_f(box[0]) / nx))
        sim.add_species(-1.0, q, (c["ppcx"], c["ppcy"]), _records(p))
        L = _laser(c, seed)
        L["start"] += shift
        sim.add_laser(type="gaussian", W0=PULSE["W0"], focus=PULSE["focus"] + shift, axis=box[1] / 2, **L)
        sim.set_moving_window()
        sim.set_device_injector(0, "step", start=c["start"])
        sim.set_smooth("binomial", c["level"], "none", 0)
        if c["graphs"]:
            sim.set_graphs(True)
        return dict(c=c, sim=sim, grids=_Grids(sim))
    if kind == "scan":
        runs, sims = _scan_table(c), []
        for k, r in enumerate(runs):
            sp = []
            for s in range(2):
                p = _plasma(r.nx[0], r.nx[1], r.ppc[0], r.ppc[1], r.uth, (1 - 2 * s) * r.uz, _gen(seed, 2 * k + s))
                sp.append((-1.0, -1.0 / (r.ppc[0] * r.ppc[1]), r.ppc, _records(p)))
            sims.append(batch.make_sim(r, sp, tile=_tile(c), sort_every=c["sort_every"]))
        return dict(c=c, runs=runs, sims=sims, batch=CudaBatch(sims), grids=[_Grids(s) for s in sims])
    if kind == "em1d":
        nx = c["nx"]
        sim = em1d_gpu.CudaSim1D(nx, nx * 0.02, 0.019, moving_window=True)
        dx = _f(_f(nx * 0.02) / nx)
        p = _plasma(nx, 1, c["ppc"], 1, 0.0, 0.0, None, i0=_f(c["start"]) / dx)
        rec = np.zeros(p["ix"].numel(), dtype=em1d_gpu.PART_DTYPE)
        rec["ix"], rec["x"] = p["ix"].cpu().numpy(), p["x"].cpu().numpy()
        sim.add_species(-1.0, -1.0 / c["ppc"], c["ppc"], rec, density=("step", c["start"], 0.0))
        L = _laser(c, seed)
        sim.add_laser(L["start"] + (nx - 1000) * 0.02, L["a0"], L["omega0"], fwhm=L["fwhm"],
                      polarization=L["polarization"])
        sim.set_smooth("compensated", c["level"])
        return dict(c=c, sim=sim)
    nx, ny = c["nx"], c["ny"]
    st, w = _adjoint_inputs(c, seed)
    sim = adjoint.AdjointSim((nx, ny), (nx * 0.1, ny * 0.1), 0.06, w.numel(), -1.0 / (c["ppcx"] * c["ppcy"]),
                             checkpoint_every=c["every"])
    host = {k: v.cpu().numpy() for k, v in st.items()}
    return dict(c=c, sim=sim, host=host, w=w.cpu().numpy())


def _adjoint_inputs(c, seed):
    """a thermal plasma whose particle weights follow a density of eight sines"""
    p = _plasma(c["nx"], c["ny"], c["ppcx"], c["ppcy"], c["uth"], 0.0, _gen(seed))
    st = {k: (v if k in ("ix", "iy") else v.double()) for k, v in p.items()}
    amps = (torch.rand(8, generator=_gen(seed, 5), device="cuda", dtype=F64) * 2 - 1) / 8
    k = 2 * math.pi * torch.arange(1, 9, device="cuda", dtype=F64) / (c["nx"] * 0.1)
    X = (st["ix"] + st["x"]) * 0.1
    w = 1 + 0.3 * (torch.sin(X[:, None] * k) * amps).sum(1)
    return st, w


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _single(*parts):
    """energies in the precision of the fields and particles they sum"""
    return torch.from_numpy(np.concatenate(parts)).float()


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind in ("em2d", "wakefield"):
        sim = state["sim"]
        sim.step(c["steps"])
        out = state["grids"].all()
        if c.get("energy"):
            out["energy"] = _single(*sim.energy())
        return out
    if kind == "scan":
        for s in state["sims"]:
            s.history_reset()
        state["batch"].step(c["steps"])
        return {"history": [torch.from_numpy(s.history()).float() for s in state["sims"]],
                "EB": [g.fields() for g in state["grids"]]}
    if kind == "report":
        sim = state["sim"]
        L, u = c["nx"] * 0.1, 6 * c["uth"]
        return {"charge": sim.charge(0),
                "x1u1": sim.phasespace(0, ("x1", "u1"), (c["pha_nx"], c["pha_nu"]), ((0.0, L), (-u, u))),
                "u2u3": sim.phasespace(0, ("u2", "u3"), (c["pha_nu"], c["pha_nu"]), ((-u, u), (-u, u)))}
    if kind == "em1d":
        sim = state["sim"]
        sim.step(c["steps"])
        emf, kin = sim.energy()
        n = c["nx"]
        return {"E": sim.E()[1:n + 1], "B": sim.B()[1:n + 1], "J": sim.J()[1:n + 1], "energy": _single(emf, kin)}
    sim, h = state["sim"], state["host"]
    sim.set_state(h["ix"], h["iy"], h["x"], h["y"], h["ux"], h["uy"], h["uz"], state["w"])
    L, kin = sim.forward(c["steps"])
    g = sim.backward()
    # the engine works in float32: its gradients and its objective in that precision
    out = {k: torch.from_numpy(v).float() for k, v in g.items()}
    out["objective"] = _single(np.array([L, kin]))
    return out


def work(case):
    """Bytes: 28-byte particle records read and written, fields read and
    written and the current once a step; flops: about 250 a particle and step
    (gather, rotation, move, deposit)."""
    c = dict(case)
    kind = c["kind"]
    if kind in ("em2d", "wakefield"):
        cells, n = c["nx"] * c["ny"], c["nx"] * c["ny"] * c["ppcx"] * c["ppcy"] * c.get("nspec", 1)
        if kind == "wakefield":
            n = int(n * (1 - c["start"] / (c["nx"] * WAKE["dx"])))
        return {"bytes": c["steps"] * (56 * n + 84 * cells), "flops": c["steps"] * (250 * n + 60 * cells)}
    if kind == "scan":
        n = sum(r.particles() for r in _scan_table(c))
        cells = sum(r.nx[0] * r.nx[1] for r in _scan_table(c))
        return {"bytes": c["steps"] * (56 * n + 84 * cells), "flops": c["steps"] * (250 * n + 60 * cells)}
    if kind == "report":
        n = c["nx"] * c["ny"] * c["ppcx"] * c["ppcy"]
        grids = 4 * (c["nx"] * c["ny"] + c["pha_nx"] * c["pha_nu"] + c["pha_nu"] ** 2)
        return {"bytes": 28 * n + grids, "flops": 60 * n}
    if kind == "em1d":
        n = int(c["nx"] * c["ppc"] * (1 - c["start"] / (c["nx"] * 0.02)))
        return {"bytes": c["steps"] * (40 * n + 84 * c["nx"]), "flops": c["steps"] * 150 * n}
    n, cells = c["nx"] * c["ny"] * c["ppcx"] * c["ppcy"], c["nx"] * c["ny"]
    # host arrays in and out once; forward, recomputed forward and reverse steps
    return {"bytes": 108 * n + 96 * cells + c["steps"] * 3 * (56 * n + 84 * cells),
            "flops": c["steps"] * 1000 * n}


# ---------------------------------------------------------------------------
# the same pass in 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """The 2-D step on grids [3, ny + 3, nx + 3] whose cell (i, j) sits at
    [j + 1, i + 1], guard cells as the step keeps them."""

    CHUNK = 1 << 22

    def __init__(self, nx, ny, dx, dy, dt, window=False, passes=((), ()), B0=None):
        self.nx, self.ny, self.dx, self.dy, self.dt = nx, ny, dx, dy, dt
        self.window, self.passes, self.B0 = window, passes, B0
        self.E = torch.zeros((3, ny + 3, nx + 3), dtype=F64, device="cuda")
        self.B, self.J = torch.zeros_like(self.E), torch.zeros_like(self.E)
        self.iter = self.moves = 0

    def at(self, i, j):
        return (j + 1) * (self.nx + 3) + i + 1

    def lerp(self, F, comp, i, j, wx, wy):
        f, k, row = F[comp].reshape(-1), self.at(i, j), self.nx + 3
        return (f[k] * (1 - wx) + f[k + 1] * wx) * (1 - wy) + (f[k + row] * (1 - wx) + f[k + row + 1] * wx) * wy

    def push(self, p, q, m_q, w=None):
        """momenta and positions of p after the step, and its current added to J"""
        i, j, x, y = p["ix"], p["iy"], p["x"], p["y"]
        lx, ly = x.detach() < 0.5, y.detach() < 0.5
        ih, jh = i - lx.long(), j - ly.long()
        xh, yh = torch.where(lx, x + 0.5, x - 0.5), torch.where(ly, y + 0.5, y - 0.5)
        E, B, t = self.E, self.B, 0.5 * self.dt / m_q
        e = torch.stack([self.lerp(E, 0, ih, j, xh, y), self.lerp(E, 1, i, jh, x, yh), self.lerp(E, 2, i, j, x, y)]) * t
        b = torch.stack([self.lerp(B, 0, i, jh, x, yh), self.lerp(B, 1, ih, j, xh, y), self.lerp(B, 2, ih, jh, xh, yh)])
        if self.B0 is not None:
            b = b + self.B0[:, None]
        u = torch.stack([p["ux"], p["uy"], p["uz"]]) + e
        u2 = (u * u).sum(0)
        g = torch.sqrt(1 + u2)
        kin = (u2 / (g + 1)).sum()
        b = b * (t / g)
        s = 2 / (1 + (b * b).sum(0))
        u = u + s * torch.linalg.cross(u + torch.linalg.cross(u, b, dim=0), b, dim=0) + e
        rg = 1 / torch.sqrt(1 + (u * u).sum(0))
        mx, my, qvz = self.dt / self.dx * rg * u[0], self.dt / self.dy * rg * u[1], q * u[2] * rg
        x1, y1 = x + mx, y + my
        di = (x1.detach() >= 1).long() - (x1.detach() < 0).long()
        dj = (y1.detach() >= 1).long() - (y1.detach() < 0).long()
        # the straight path cut where it meets a cell edge: up to three pieces
        one = torch.ones_like(mx)
        tx = torch.where(di != 0, ((di > 0).to(F64) - x) / torch.where(di != 0, mx, one), one)
        ty = torch.where(dj != 0, ((dj > 0).to(F64) - y) / torch.where(dj != 0, my, one), one)
        first, last = torch.minimum(tx, ty), torch.maximum(tx, ty)
        xf, yf = (tx <= ty).long(), (ty < tx).long()
        cuts = [(torch.zeros_like(mx), first, 0 * di, 0 * dj), (first, last, di * xf, dj * yf), (last, one, di, dj)]
        J = self.J.reshape(-1)
        plane, row = (self.nx + 3) * (self.ny + 3), self.nx + 3
        qw = one if w is None else w
        for n, (a, z, ci, cj) in enumerate(cuts):
            f = (z - a) * qw
            x0, xe, y0, ye = x + mx * a - ci, x + mx * z - ci, y + my * a - cj, y + my * z - cj
            k = self.at(i + ci, j + cj)
            sel = slice(None)
            if n:  # most particles stay in their cell
                sel = torch.nonzero((di != 0) | (dj != 0))[:, 0]
                f, x0, xe, y0, ye, k = f[sel], x0[sel], xe[sel], y0[sel], ye[sel], k[sel]
            jx, jy = q * self.dx / self.dt * mx[sel] * f, q * self.dy / self.dt * my[sel] * f
            qz = 0.5 * qvz[sel] * f
            ym, xm = 0.5 * (y0 + ye), 0.5 * (x0 + xe)
            J = J.index_add(0, torch.cat([k, k + row]), torch.cat([jx * (1 - ym), jx * ym]))
            J = J.index_add(0, plane + torch.cat([k, k + 1]), torch.cat([jy * (1 - xm), jy * xm]))
            for cx in (0, 1):
                sx0, sx1 = (x0, xe) if cx else (1 - x0, 1 - xe)
                for cy in (0, 1):
                    sy0, sy1 = (y0, ye) if cy else (1 - y0, 1 - ye)
                    J = J.index_add(0, 2 * plane + k + cx + cy * row,
                                    qz * (sx0 * sy0 + sx1 * sy1 + (sx0 * sy1 - sx1 * sy0) / 2))
        self.J = J.reshape(self.J.shape)
        i, j = i + di, (j + dj) % self.ny
        if not self.window:
            i = i % self.nx
        return dict(ix=i, iy=j, x=x1 - di, y=y1 - dj, ux=u[0], uy=u[1], uz=u[2]), kin

    def update_current(self):
        J, nx, ny = self.J, self.nx, self.ny
        if not self.window:
            J[:, :, 0:3] += J[:, :, nx:nx + 3]
            J[:, :, nx:nx + 3] = J[:, :, 0:3]
        J[:, 0:3] += J[:, ny:ny + 3]
        J[:, ny:ny + 3] = J[:, 0:3]
        for sa, sb in self.passes[0]:
            J[:, 1:ny + 1, 1:nx + 1] = (sa * (J[:, 1:ny + 1, 0:nx] + J[:, 1:ny + 1, 2:nx + 2])
                                        + sb * J[:, 1:ny + 1, 1:nx + 1])
            if not self.window:
                J[:, 1:ny + 1, 0] = J[:, 1:ny + 1, nx]
                J[:, 1:ny + 1, nx + 1:nx + 3] = J[:, 1:ny + 1, 1:3].clone()
        # the y passes leave the x guard columns as they are, and the first reads the y guard rows unfiltered
        for sa, sb in self.passes[1]:
            J[:, 1:ny + 1, 1:nx + 1] = sa * (J[:, 0:ny, 1:nx + 1] + J[:, 2:ny + 2, 1:nx + 1]) + sb * J[:, 1:ny + 1, 1:nx + 1]
            J[:, 0] = J[:, ny]
            J[:, ny + 1:ny + 3] = J[:, 1:3].clone()

    def guards(self, F):
        nx, ny = self.nx, self.ny
        if not self.window:
            F = torch.cat([F[:, :, nx:nx + 1], F[:, :, 1:nx + 1], F[:, :, 1:3]], dim=2)
        return torch.cat([F[:, ny:ny + 1], F[:, 1:ny + 1], F[:, 1:3]], dim=1)

    def half_b(self, E, B):
        hx, hy, nx, ny = 0.5 * self.dt / self.dx, 0.5 * self.dt / self.dy, self.nx, self.ny
        a, r, d = (E[:, 0:ny + 2, 0:nx + 2], E[:, 0:ny + 2, 1:nx + 3], E[:, 1:ny + 3, 0:nx + 2])
        new = B.clone()
        new[0, 0:ny + 2, 0:nx + 2] -= hy * (d[2] - a[2])
        new[1, 0:ny + 2, 0:nx + 2] += hx * (r[2] - a[2])
        new[2, 0:ny + 2, 0:nx + 2] += hy * (d[0] - a[0]) - hx * (r[1] - a[1])
        return new

    def advance_fields(self):
        cx, cy, nx, ny, dt = self.dt / self.dx, self.dt / self.dy, self.nx, self.ny, self.dt
        B = self.half_b(self.E, self.B)
        a, l, d = B[:, 1:ny + 3, 1:nx + 3], B[:, 1:ny + 3, 0:nx + 2], B[:, 0:ny + 2, 1:nx + 3]
        E = self.E.clone()
        J = self.J[:, 1:ny + 3, 1:nx + 3]
        E[0, 1:ny + 3, 1:nx + 3] += cy * (a[2] - d[2]) - dt * J[0]
        E[1, 1:ny + 3, 1:nx + 3] += -cx * (a[2] - l[2]) - dt * J[1]
        E[2, 1:ny + 3, 1:nx + 3] += cx * (a[1] - l[1]) - cy * (a[0] - d[0]) - dt * J[2]
        B = self.half_b(E, B)
        self.E, self.B = self.guards(E), self.guards(B)
        self.iter += 1

    def moves_now(self):
        return self.window and np.float32(self.iter) * np.float32(self.dt) > np.float32(self.dx) * np.float32(self.moves + 1)

    def shift_fields(self):
        for F in (self.E, self.B):
            F[:, :, :-1] = F[:, :, 1:].clone()
            F[:, :, -3:] = 0
        self.moves += 1

    def step(self, species, column=None):
        """[(q, particles)] after one step (charge over mass -1), and their kinetic energies"""
        self.J = torch.zeros_like(self.E)
        out, kins = [], []
        for q, p in species:
            parts, kin = [], 0.0
            for a in range(0, max(p["ix"].numel(), 1), self.CHUNK):
                new, k = self.push({n: v[a:a + self.CHUNK] for n, v in p.items()}, q, -1.0)
                parts.append(new)
                kin = kin + k
            p = {n: torch.cat([v[n] for v in parts]) for n in p}
            kins.append(-q * kin * self.dx * self.dy)
            out.append((q, p))
        self.update_current()
        self.advance_fields()
        if self.moves_now():
            self.shift_fields()
            for k, (q, p) in enumerate(out):
                p["ix"] = p["ix"] - 1
                out[k] = (q, {n: torch.cat([v, column[n]]) for n, v in p.items()})
        if self.window:
            for k, (q, p) in enumerate(out):
                keep = (p["ix"] >= 0) & (p["ix"] < self.nx)
                out[k] = (q, {n: v[keep] for n, v in p.items()})
        return out, kins

    def interior(self, F):
        return F[:, 1:self.ny + 1, 1:self.nx + 1]

    def field_energy(self):
        return 0.5 * self.dx * self.dy * torch.cat([(self.interior(F) ** 2).sum((1, 2)) for F in (self.E, self.B)])


def _double(p):
    return {k: (v.long() if k in ("ix", "iy") else v.double()) for k, v in p.items()}


def _passes(kind, level):
    """the filter's (side, middle) weights, pass by pass"""
    p = [(0.25, 0.5)] * level if kind != "none" else []
    if kind == "compensated":
        b = (4.0 + 2.0 * level) / level
        p.append((-1.0 / (b - 2.0), b / (b - 2.0)))
    return tuple(p)


def _pulse(L, z):
    """longitudinal envelope, sin^2 up and down over the FWHM"""
    u = (z - L["start"]) / L["fwhm"]
    e = torch.sin(0.5 * math.pi * u) ** 2
    return torch.where((u <= 0) & (u > -2), e, torch.zeros_like(e))


def _exact2d(c, seed):
    nx, ny = c["nx"], c["ny"]
    dx, dy = _f(_f(nx * 0.1) / np.float32(nx)), _f(_f(ny * 0.1) / np.float32(ny))
    p = _passes(c["filter"], c["level"])
    B0 = torch.tensor([0.0, 0.0, _f(c["ext"])], dtype=F64, device="cuda") if c["ext"] else None
    X = _Exact(nx, ny, dx, dy, _f(c["dt"]), passes=(p, p), B0=B0)
    sp = [(_f(q), _double(p)) for q, p in _species(c, seed)]
    for _ in range(c["steps"]):
        sp, kin = X.step(sp)
    out = {"EB": torch.cat([X.interior(X.E), X.interior(X.B)]), "J": X.interior(X.J)}
    if c["energy"]:
        out["energy"] = torch.cat([X.field_energy(), torch.stack(kin)])
    return out


def _exact_wakefield(c, seed):
    nx, ny = c["nx"], c["ny"]
    box, shift = _window(c)
    dx, dy = _f(_f(box[0]) / np.float32(nx)), _f(_f(box[1]) / np.float32(ny))
    X = _Exact(nx, ny, dx, dy, _f(WAKE["dt"]), window=True, passes=(_passes("binomial", c["level"]), ()))
    L = _laser(c, seed)
    L["start"] += shift
    amp, cp, sp = L["omega0"] * L["a0"], math.cos(L["polarization"]), math.sin(L["polarization"])
    z = torch.arange(nx, device="cuda", dtype=F64)[None, :] * dx
    r = torch.arange(ny, device="cuda", dtype=F64)[:, None] * dy - box[1] / 2

    def gauss(zz, rr):
        d, zr = zz - (PULSE["focus"] + shift), L["omega0"] * PULSE["W0"] ** 2 / 2
        w = zr * zr / (zr * zr + d * d)
        ph = L["omega0"] * (d + rr * rr * d / (zr * zr + d * d)) - torch.atan2(d, torch.full_like(d, zr))
        return torch.sqrt(torch.sqrt(w)) * torch.exp(-rr * rr * w / PULSE["W0"] ** 2) * torch.cos(ph)

    a, a2 = amp * _pulse(L, z), amp * _pulse(L, z + dx / 2)
    rows, cols = slice(1, ny + 1), slice(1, nx + 1)
    X.E[1, rows, cols] = a * gauss(z, r + dy / 2) * cp
    X.E[2, rows, cols] = a * gauss(z, r) * sp
    X.B[1, rows, cols] = -a2 * gauss(z + dx / 2, r) * sp
    X.B[2, rows, cols] = a2 * gauss(z + dx / 2, r + dy / 2) * cp
    # no divergence: Ex and Bx summed from the right (guard rows are still zero)
    ex = dx / dy * (X.E[1, rows, 2:nx + 2] - X.E[1, 0:ny, 2:nx + 2])
    bx = dx / dy * (X.B[1, 2:ny + 2, cols] - X.B[1, rows, cols])
    X.E[0, rows, cols] = ex.flip(1).cumsum(1).flip(1)
    X.B[0, rows, cols] = bx.flip(1).cumsum(1).flip(1)
    X.E, X.B = X.guards(X.E), X.guards(X.B)
    ppc = (c["ppcx"], c["ppcy"])
    p = _plasma(nx, ny, *ppc, 0.0, 0.0, None, i0=_f(c["start"]) / dx)
    col = _double(_plasma(1, ny, *ppc, 0.0, 0.0, None))
    col["ix"] = col["ix"] + nx - 1
    sp = [(_f(-1.0 / (ppc[0] * ppc[1])), _double(p))]
    for _ in range(c["steps"]):
        sp, _kin = X.step(sp, col)
    return {"EB": torch.cat([X.interior(X.E), X.interior(X.B)]), "J": X.interior(X.J)}


def _exact_scan(c, seed):
    rows, fields = [], []
    for k, r in enumerate(_scan_table(c)):
        nx, ny = r.nx
        dx, dy = (_f(_f(r.box[a]) / np.float32(r.nx[a])) for a in (0, 1))
        X = _Exact(nx, ny, dx, dy, _f(r.dt))
        sp = [(_f(-1.0 / (r.ppc[0] * r.ppc[1])),
               _double(_plasma(nx, ny, r.ppc[0], r.ppc[1], r.uth, (1 - 2 * s) * r.uz, _gen(seed, 2 * k + s))))
              for s in range(2)]
        hist = []
        for _ in range(c["steps"]):
            sp, kin = X.step(sp)
            hist.append(torch.cat([X.field_energy(), torch.stack(kin)]))
        rows.append(torch.stack(hist))
        fields.append(torch.cat([X.interior(X.E), X.interior(X.B)]))
    return {"history": rows, "EB": fields}


def _bilinear(out, i, j, wx, wy, v, drop):
    """v shared among the four corners of (i, j) of out [n2, n1]"""
    n2, n1 = out.shape
    for cx in (0, 1):
        for cy in (0, 1):
            a, b = i + cx, j + cy
            part = v * (wx if cx else 1 - wx) * (wy if cy else 1 - wy)
            if drop:
                ok = (a >= 0) & (a < n1) & (b >= 0) & (b < n2)
                a, b, part = a[ok], b[ok], part[ok]
            out.view(-1).index_add_(0, b * n1 + a, part)


def _exact_report(c, seed):
    (q, p), = _species(c, seed)
    nx, ny = c["nx"], c["ny"]
    p32 = p
    p = _double(p)
    v = torch.full_like(p["x"], _f(q))
    rho = torch.zeros((ny + 1, nx + 1), dtype=F64, device="cuda")
    _bilinear(rho, p["ix"], p["iy"], p["x"], p["y"], v, False)
    rho[:, 0] += rho[:, nx]
    rho[0] += rho[ny]
    L, u = c["nx"] * 0.1, 6 * c["uth"]
    dx = _f(_f(L) / np.float32(nx))

    def density(a, b, n, lo, hi):
        pos = [(w - _f(lo[k])) * (n[k] / (_f(hi[k]) - _f(lo[k]))) for k, w in enumerate((a, b))]
        at = [(w + 0.5).trunc().long() for w in pos]
        out = torch.zeros((n[1], n[0]), dtype=F64, device="cuda")
        _bilinear(out, at[0], at[1], pos[0] - at[0] + 0.5, pos[1] - at[1] + 0.5, v, True)
        return out

    x1 = (p32["ix"] + p["x"]) * dx
    return {"charge": rho, "x1u1": density(x1, p["ux"], (c["pha_nx"], c["pha_nu"]), (0.0, -u), (L, u)),
            "u2u3": density(p["uy"], p["uz"], (c["pha_nu"], c["pha_nu"]), (-u, -u), (u, u))}


def _exact1d(c, seed):
    nx, dt = c["nx"], _f(0.019)
    dx = _f(_f(nx * 0.02) / np.float32(nx))
    E = torch.zeros((3, nx + 3), dtype=F64, device="cuda")
    B = torch.zeros_like(E)
    L = _laser(c, seed)
    L["start"] += (nx - 1000) * 0.02
    amp, cp, sp = L["omega0"] * L["a0"], math.cos(L["polarization"]), math.sin(L["polarization"])
    z = torch.arange(nx, device="cuda", dtype=F64) * dx
    a, a2 = amp * _pulse(L, z), amp * _pulse(L, z + dx / 2)
    c1, c2 = torch.cos(L["omega0"] * z), torch.cos(L["omega0"] * (z + dx / 2))
    E[1, 1:nx + 1], E[2, 1:nx + 1] = a * c1 * cp, a * c1 * sp
    B[1, 1:nx + 1], B[2, 1:nx + 1] = -a2 * c2 * sp, a2 * c2 * cp
    p = _double(_plasma(nx, 1, c["ppc"], 1, 0.0, 0.0, None, i0=_f(c["start"]) / dx))
    lat = ((torch.arange(c["ppc"], device="cuda") + 0.5) / c["ppc"]).float().double()
    i, x, u = p["ix"], p["x"], torch.stack([p["ux"], p["uy"], p["uz"]])
    q, t = _f(-1.0 / c["ppc"]), -0.5 * dt
    moves = 0

    def mid(F, k, cell, w):
        return F[k][cell + 1] * (1 - w) + F[k][cell + 2] * w

    def half_b():
        B[1, 0:nx + 2] += 0.5 * dt / dx * (E[2, 1:nx + 3] - E[2, 0:nx + 2])
        B[2, 0:nx + 2] -= 0.5 * dt / dx * (E[1, 1:nx + 3] - E[1, 0:nx + 2])

    for n in range(c["steps"]):
        low = (x < 0.5).long()
        h, w = i - low, torch.where(low > 0, x + 0.5, x - 0.5)
        e = torch.stack([mid(E, 0, h, w), mid(E, 1, i, x), mid(E, 2, i, x)]) * t
        b = torch.stack([mid(B, 0, i, x), mid(B, 1, h, w), mid(B, 2, h, w)])
        u = u + e
        u2 = (u * u).sum(0)
        g = torch.sqrt(1 + u2)
        kin = (u2 / (1 + g)).sum()
        b = b * (t / g)
        s = 2 / (1 + (b * b).sum(0))
        u = u + s * torch.linalg.cross(u + torch.linalg.cross(u, b, dim=0), b, dim=0) + e
        rg = 1 / torch.sqrt(1 + (u * u).sum(0))
        m = dt / dx * rg * u[0]
        x1 = x + m
        di = (x1 >= 1).long() - (x1 < 0).long()
        one = torch.ones_like(m)
        cut = torch.where(di != 0, ((di > 0).to(F64) - x) / torch.where(di != 0, m, one), one)
        J = torch.zeros_like(E)
        for f, x0, xe, cell in ((cut, x, x + m * cut, i), (1 - cut, x + m * cut - di, x1 - di, i + di)):
            J[0].index_add_(0, cell + 1, q * dx / dt * m * f)
            for k in (1, 2):
                v = 0.5 * q * u[k] * rg * f
                J[k].index_add_(0, cell + 1, v * ((1 - x0) + (1 - xe) + (xe - x0) / 2))
                J[k].index_add_(0, cell + 2, v * (x0 + xe + (x0 - xe) / 2))
        for sa, sb in _passes("compensated", c["level"]):
            J[:, 1:nx + 1] = sa * (J[:, 0:nx] + J[:, 2:nx + 2]) + sb * J[:, 1:nx + 1]
        x, i = x1 - di, i + di
        half_b()
        E[0, 1:nx + 3] -= dt * J[0, 1:nx + 3]
        E[1, 1:nx + 3] += -dt / dx * (B[2, 1:nx + 3] - B[2, 0:nx + 2]) - dt * J[1, 1:nx + 3]
        E[2, 1:nx + 3] += dt / dx * (B[1, 1:nx + 3] - B[1, 0:nx + 2]) - dt * J[2, 1:nx + 3]
        half_b()
        if np.float32(n + 1) * np.float32(dt) > np.float32(dx) * np.float32(moves + 1):
            moves += 1
            for F in (E, B):
                F[:, :-1] = F[:, 1:].clone()
                F[:, -3:] = 0
            i = torch.cat([i - 1, torch.full((c["ppc"],), nx - 1, device="cuda")])
            x = torch.cat([x, lat])
            u = torch.cat([u, torch.zeros((3, c["ppc"]), dtype=F64, device="cuda")], dim=1)
        keep = (i >= 0) & (i < nx)
        i, x, u = i[keep], x[keep], u[:, keep]
    cells = slice(1, nx + 1)
    emf = 0.5 * dx * torch.cat([(F[:, cells] ** 2).sum(1) for F in (E, B)])
    return {"E": E[:, cells].T, "B": B[:, cells].T, "J": J[:, cells].T,
            "energy": torch.cat([emf, (-q * kin * dx)[None]])}


def _exact_adjoint(c, seed):
    from torch.utils.checkpoint import checkpoint

    nx, ny = c["nx"], c["ny"]
    st, w = _adjoint_inputs(c, seed)
    X = _Exact(nx, ny, 0.1, 0.1, 0.06)
    names = ("x", "y", "ux", "uy", "uz")
    leaf = {k: st[k].clone().requires_grad_() for k in names}
    w = w.clone().requires_grad_()
    E0 = torch.zeros((3, ny, nx), dtype=F64, device="cuda", requires_grad=True)
    B0 = torch.zeros((3, ny, nx), dtype=F64, device="cuda", requires_grad=True)
    q = -1.0 / (c["ppcx"] * c["ppcy"])

    def pad(F):
        return torch.nn.functional.pad(F, (1, 2, 1, 2), mode="circular")

    def step(E, B, i, j, x, y, ux, uy, uz, w):
        X.E, X.B = pad(E), pad(B)
        X.J = torch.zeros_like(X.E)
        p, kin = X.push(dict(ix=i, iy=j, x=x, y=y, ux=ux, uy=uy, uz=uz), q, -1.0, w)
        J = X.J  # folded onto the periodic cells
        J = J[:, :, 1:nx + 1] + torch.nn.functional.pad(J[:, :, nx + 1:nx + 3], (0, nx - 2)) \
            + torch.nn.functional.pad(J[:, :, 0:1], (nx - 1, 0))
        J = J[:, 1:ny + 1] + torch.nn.functional.pad(J[:, ny + 1:ny + 3], (0, 0, 0, ny - 2)) \
            + torch.nn.functional.pad(J[:, 0:1], (0, 0, ny - 1, 0))
        X.J = pad(J)
        X.advance_fields()
        return (X.interior(X.E), X.interior(X.B), p["ix"], p["iy"], p["x"], p["y"], p["ux"], p["uy"], p["uz"])

    s = (E0, B0, st["ix"].long(), st["iy"].long(), *[leaf[k] for k in names])
    for _ in range(c["steps"]):
        s = checkpoint(step, *s, w, use_reentrant=False)
    Lx = 0.5 * 0.1 * 0.1 * ((s[0] ** 2).sum() + (s[1] ** 2).sum())
    Lx.backward()
    out = {k: leaf[k].grad for k in names}
    out.update(w=w.grad, E=E0.grad, B=B0.grad, objective=None)
    return out


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "em2d":
        return _exact2d(c, seed)
    if kind == "wakefield":
        return _exact_wakefield(c, seed)
    if kind == "scan":
        return _exact_scan(c, seed)
    if kind == "report":
        return _exact_report(c, seed)
    if kind == "em1d":
        return _exact1d(c, seed)
    return _exact_adjoint(c, seed)
