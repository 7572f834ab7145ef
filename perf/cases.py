"""Timed cases of the framework: the steps that a simulation spends its time in.

A case is one scene (a channel, a suspension, a Couette cell, a constriction,
a box of plain fluid, an ensemble of suspensions) stepped a few times through
one of the public entry points:

* ``fused``    -- ``FusedSystem``, host-driven steps (the default);
* ``captured`` -- ``FusedSystem(graph=True)``, each step one CUDA graph;
* ``ensemble`` -- ``Ensemble``: many independent systems in the same launches;
* ``dropin``   -- ``host.ParticleSystem``: GPUCell's own call sequence through
  the 20 boundary entry points on buffers that the caller owns.

The seed of a state draws the fluid's displacements from its lattice and the
thermal velocities of every moving particle; the scene itself (walls, cells,
lattice) follows from the case and is built once per process.  A pass hands
the simulation its state (device arrays in original order; the drop-in's
caller restores its own buffers), advances it by ``steps`` timesteps and
takes it back whole, in original particle order, as a program does that
couples the simulation to another one or branches trajectories from a state.
Two states are handed over in turn, so that every pass of the library-owned
simulations re-sorts and rebuilds the neighbour lists once, in its first
step: one rebuild per 12 to 16 steps (a running suspension needs one per 8
to 10).  Positions come back unwrapped (position + crossings times box
length), as a program that tracks particles or membranes uses them.  The
Morse force ends at its cut-off with a jump, so a pair there counts or not by
the last bit of a position; the scene with tens of thousands of aggregating
vertices returns deformation and aggregation force as one sum, in which that
is lost.

``exact`` is the method in 64 bits, in plain torch: integration, densities,
SDPD pair forces with their Philox pair noise, wall repulsion and no-slip
walls, membrane mechanics and Morse aggregation.
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import functools
import math

import numpy as np
import torch

from gpucell_gb300 import _lib, generator
from gpucell_gb300.fused import Ensemble, FusedSystem
from gpucell_gb300.host import ParticleSystem

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
DX = 1.0 / 3.0


def listed():
    return [
        # The smallest simulation the tests use (every particle type, one
        # small cell): a parameter study's or a tutorial's channel, where
        # launches and latency count.
        dict(name="channel_6k", api="fused", scene="channel", nx=24, ny=12, nz=12, ncells=1, subdiv=2, b1=1, noise=True,
             steps=16),
        # A small channel with one red cell in captured steps, the mode for
        # small systems that run long between two outputs.
        dict(name="channel_24k_captured", api="captured", scene="channel", nx=42, ny=20, nz=22, ncells=1, subdiv=3, b1=1,
             noise=True, steps=16),
        # The 65,536-fluid Poiseuille channel with a 642-vertex cell, noise
        # off: validation runs against the analytic profile.
        dict(name="channel_78k_quiet", api="fused", scene="channel", nx=64, ny=32, nz=32, ncells=1, subdiv=3, b1=0,
             noise=False, steps=16),
        # Plain fluid in a box whose sides fit no power of two: equilibration
        # and viscosity measurements.
        dict(name="fluid_152k", api="fused", scene="fluid", nx=61, ny=47, nz=53, ncells=0, subdiv=3, b1=0, noise=True,
             steps=16),
        # Flow through a 2:1 constriction with walls of both kinds, 25 cells.
        dict(name="constriction_488k", api="fused", scene="constriction", nx=140, ny=96, nz=36, ncells=25, subdiv=3, b1=1,
             noise=True, steps=16),
        # Cells of 2562 vertices in Couette flow with Morse aggregation.
        dict(name="sheared_350k", api="fused", scene="sheared", nx=68, ny=64, nz=68, ncells=16, subdiv=4, b1=0, noise=True,
             steps=16),
        # The half-million-particle red-cell suspension of the small benchmark.
        dict(name="suspension_524k", api="fused", scene="suspension", nx=128, ny=64, nz=64, ncells=25, subdiv=4, b1=0,
             noise=True, steps=16),
        # The benchmark's suspension: 4.2 million particles, 200 cells.
        dict(name="suspension_4m", api="fused", scene="suspension", nx=128, ny=64, nz=64, ncells=25, subdiv=4, b1=0,
             noise=True, steps=12, tiles=2),
        # Sixteen independent suspensions of uneven size in one ensemble.
        dict(name="ensemble_16", api="ensemble", scene="suite", nsys=16, n_low=8000, n_high=60000, b1=0, noise=True,
             steps=12),
        # GPUCell's call sequence on the caller's buffers: the channel with a
        # cell and walls of both kinds, ...
        dict(name="dropin_channel_83k", api="dropin", scene="channel", nx=64, ny=32, nz=32, ncells=1, subdiv=3, b1=1,
             noise=True, steps=5),
        # ... a rouleau of four cells in Couette flow with aggregation, ...
        dict(name="dropin_couette_80k", api="dropin", scene="couette", nx=64, ny=32, nz=32, ncells=4, subdiv=3, b1=0,
             noise=True, steps=5),
        # ... and a million-particle suspension (one step: the boundary keeps
        # FP32 positions, whose last bit moves the stiff membranes' forces).
        dict(name="dropin_suspension_1m", api="dropin", scene="suspension", nx=128, ny=64, nz=128, ncells=50, subdiv=4,
             b1=0, noise=True, steps=1),
    ]


def draw(rng):
    """One more case of the same ranges: any entry point, 6 thousand to a
    million particles, sides of any parity."""
    api = rng.choice(["fused", "fused", "fused", "captured", "ensemble", "dropin", "dropin"])
    if api == "ensemble":
        low = rng.randint(6000, 12000)
        return dict(api=api, scene="suite", nsys=rng.randint(4, 24), n_low=low,
                    n_high=int(low * math.exp(rng.uniform(0.3, 2.0))), b1=0, noise=rng.random() < 0.8,
                    steps=rng.randint(5, 9))
    scene = rng.choice(["channel", "channel", "fluid", "suspension", "suspension", "couette", "sheared", "constriction"])
    top = {"captured": 3.0e5, "dropin": 5.0e5}.get(api, 1.0e6)
    n = math.exp(rng.uniform(math.log(6.0e3), math.log(top)))
    side = (n / 2.0) ** (1.0 / 3.0)
    least = {"channel": 12, "fluid": 14, "suspension": 22, "couette": 24, "sheared": 48, "constriction": 24}[scene]

    def a_side(mean):
        return max(least, int(round(mean * math.exp(rng.uniform(-0.2, 0.2)))))

    case = dict(api=api, scene=scene, nx=a_side(2.0 * side), ny=a_side(side), nz=a_side(side), ncells=0, subdiv=3,
                b1=rng.choice([0, 1]), noise=rng.random() < 0.75, steps=rng.randint(8, 16))
    if api == "dropin":
        case["steps"] = rng.randint(2, 5) if scene in ("channel", "fluid", "couette") else 1
    vol = case["nx"] * case["ny"] * case["nz"] * DX ** 3
    if scene == "channel":
        if min(case["ny"], case["nz"]) < 20:
            case["subdiv"] = 2
        case["ncells"] = rng.choice([0, 1])
    elif scene == "suspension":
        case["ncells"] = max(1, int(rng.uniform(0.02, 0.2) * vol / 28.0))
    elif scene == "couette":
        case["ncells"] = rng.choice([1, 2])
    elif scene == "sheared":
        case["subdiv"] = 4
        case["ncells"] = max(1, int(rng.uniform(0.01, 0.06) * vol / 94.0))
    elif scene == "constriction":
        case["ny"] = max(case["ny"], 60)
        case["nz"] = max(case["nz"], 24)
        case["nx"] = max(case["nx"], 60)
        case["b1"], case["ncells"] = 1, rng.choice([0, 1, 2, 4])
    return case


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
def _tiled(cfg, k):
    """A periodic suspension repeated k times along each axis."""
    if k == 1:
        return cfg
    b = cfg.bbox.astype(np.float64)
    L = b[1::2] - b[0::2]
    shifts = [np.array([i, j, l]) * L for i in range(k) for j in range(k) for l in range(k)]
    nf, m = cfg.n_fluid, len(shifts)
    coor = np.concatenate([cfg.coor[:nf] + s.astype(np.float32) for s in shifts]
                          + [cfg.coor[nf:] + s.astype(np.float32) for s in shifts]).astype(np.float32)
    rep = lambda a, step: np.concatenate([a + i * step for i in range(m)])
    edge_step = np.array([cfg.ncp] * 4 + [cfg.ntri] * 2, np.int32)
    bbox = b.copy()
    bbox[1::2] = b[0::2] + k * L
    return dataclasses.replace(
        cfg, bbox=bbox.astype(np.float32), n_fluid=nf * m, coor=coor, velhalf=np.zeros_like(coor), ncell=cfg.ncell * m,
        npar=np.tile(cfg.npar, m), ntri_cell=np.tile(cfg.ntri_cell, m), tri=rep(cfg.tri, np.int32(cfg.ncp)),
        edge=rep(cfg.edge, edge_step), betri=rep(cfg.betri, np.int32(cfg.ntri)),
        celltab=rep(cfg.celltab, np.int32(cfg.ncell)), cell_type=np.tile(cfg.cell_type, m))


@functools.lru_cache(maxsize=2)
def _scene(key):
    """The configurations of a case (one, or the systems of an ensemble)."""
    c = dict(key)
    if c["scene"] == "suite":
        return generator.ensemble_suite(nsys=c["nsys"], n_range=(c["n_low"], c["n_high"]))
    s = dict(nx=c["nx"], ny=c["ny"], nz=c["nz"])
    if c["scene"] == "channel":
        fits = 0.85 * min(c["ny"], c["nz"]) * DX
        return [generator.channel(**s, b1_layers=c["b1"], cell_subdiv=c["subdiv"] if c["ncells"] else -1,
                                  cell_diameter=min(8.0 / 1.5, fits) if c["subdiv"] > 2 else min(3.0, fits))]
    if c["scene"] == "fluid":
        return [generator.suspension(**s, ncells=0)]
    if c["scene"] == "suspension":
        d = dict(diameter=8.0 / 1.5) if c["subdiv"] == 3 else {}
        return [_tiled(generator.suspension(**s, ncells=c["ncells"], subdiv=c["subdiv"], **d), c.get("tiles", 1))]
    if c["scene"] == "couette":
        return [generator.couette(**s, ncells=c["ncells"], subdiv=c["subdiv"],
                                  cell_diameter=min(8.0 / 1.5, 0.45 * c["ny"] * DX, 0.9 * c["nz"] * DX))]
    if c["scene"] == "sheared":
        return [generator.sheared_suspension(**s, ncells=c["ncells"], subdiv=c["subdiv"])]
    return [generator.constriction(**s, b1_layers=c["b1"], ncells=c["ncells"], subdiv=c["subdiv"], layout="random")]


def _configs(case):
    return _scene(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "api", "noise", "steps"))))


def _inputs(case, seed, which=0):
    """Per system of the case: its configuration with the fluid displaced
    from the lattice, and the thermal velocities of its moving particles
    (`which`: the first or the second of the states handed over in turn)."""
    out = []
    for k, cfg in enumerate(_configs(case)):
        rng = np.random.default_rng([seed, k, which])
        fl, me = cfg.n_b1 + cfg.n_b2, cfg.n_cell_start
        coor = cfg.coor.copy()
        coor[fl:me] += (rng.random((cfg.n_fluid, 3), np.float32) - np.float32(0.5)) * np.float32(0.2 * DX)
        vel = np.zeros_like(coor)
        vel[fl:] = rng.standard_normal((cfg.n - fl, 3), np.float32) * np.float32(math.sqrt(cfg.phys.temp / cfg.phys.mass))
        # a displaced particle may have left the box at a periodic face
        for a in range(3):
            lo, hi = cfg.bbox[2 * a], cfg.bbox[2 * a + 1]
            if cfg.pmask >> a & 1:
                x = coor[fl:me, a]
                x[x < lo] += hi - lo
                x[x >= hi] -= hi - lo
        out.append((dataclasses.replace(cfg, coor=coor), vel))
    return out


# ---------------------------------------------------------------------------
# Passes
# ---------------------------------------------------------------------------
_CELLS = ("area", "vol", "defforce", "aggforce", "trinordir", "tricenter", "pararea")


def _lengths(cfg):
    """Box lengths on the periodic axes (0 elsewhere)."""
    return torch.as_tensor((cfg.bbox[1::2] - cfg.bbox[0::2]) * np.float32([cfg.pmask >> a & 1 for a in range(3)]))[None]


def _ptr(t):
    return C.c_void_p(t.data_ptr() if t is not None else 0)


def prepare(case, seed):
    cfgs = _configs(case)
    z = lambda *shape, dt=torch.float32: torch.zeros(shape, dtype=dt, device=DEVICE)
    if case["api"] == "dropin":
        (cfg, vel), = _inputs(case, seed)
        ps = ParticleSystem(cfg, device=DEVICE, noise=case["noise"])
        ps.set_state(vel=vel)
        keep = ("TotalCoor", "Velrhop", "VelHalf", "TotalForce", "SortPart", "nThroBound")
        return dict(case=case, system=ps, lengths=_lengths(cfgs[0]).to(DEVICE), start={k: ps.d[k].clone() for k in keep})
    n, ncell = sum(c.n for c in cfgs), sum(c.ncell for c in cfgs)
    ntri, ncp = sum(c.ntri for c in cfgs), sum(c.ncp for c in cfgs)
    if case["api"] == "ensemble":
        fs = Ensemble(cfgs, noise=case["noise"])
        lengths = torch.cat([_lengths(c).expand(c.n, 3) for c in cfgs]).to(DEVICE)
    else:
        fs = FusedSystem(cfgs[0], noise=case["noise"], graph=case["api"] == "captured")
        lengths = _lengths(cfgs[0]).to(DEVICE)
    up = lambda arrays: torch.as_tensor(np.concatenate(arrays), device=DEVICE)
    start = []
    for which in (0, 1):
        inputs = _inputs(case, seed, which)
        start.append([up([c.coor for c, _ in inputs]), up([v for _, v in inputs]), up([c.velhalf for c in cfgs]), z(n, 3),
                      z(n, 3, dt=torch.int32)])
    cells = dict(zip(_CELLS, (z(ncell), z(ncell), z(ncp, 3), z(ncp, 3), z(ntri, 3), z(ntri, 3), z(ncp)))) if ncell else {}
    return dict(case=case, system=fs, lengths=lengths, start=start, passes=0, pos=z(n, 3), vel=z(n, 3), rho=z(n), press=z(n),
                force=z(n, 3), nthro=z(n, 3, dt=torch.int32), cells=cells)


def _membrane(case, cells):
    if case["scene"] != "sheared":
        return cells
    return dict({k: v for k, v in cells.items() if k != "aggforce"}, defforce=cells["defforce"] + cells["aggforce"])


def run(state):
    case, s = state["case"], state["system"]
    if case["api"] == "dropin":
        d = s.d
        for k, t in state["start"].items():
            d[k].copy_(t)
        _lib.call("gc_set_step", -1)
        for _ in range(case["steps"]):
            s.update(1)
        if s.has_cells:
            slot = d["CurPos"].long()
        else:
            slot = torch.empty_like(d["SortPart"], dtype=torch.long)
            slot[d["SortPart"].long()] = torch.arange(s.n, device=DEVICE)
        vr = d["Velrhop"][slot]
        pos = d["TotalCoor"][slot]
        if s.has_cells:   # GPUCell sorts the crossing counts with the particles only where there are cells
            pos = pos + d["nThroBound"][slot] * state["lengths"]
        out = dict(pos=pos, vel=vr[:, :3], rho=vr[:, 3], press=d["Press"][slot], force=d["TotalForce"][slot])
        if s.has_cells:
            out.update(_membrane(case, dict(
                area=d["Area"], vol=d["Vol"], defforce=d["DefForce"], aggforce=d["AggForce"], trinordir=d["TriNorDir"],
                tricenter=d["TriCenter"], pararea=d["ParArea"])))
        return out
    _lib.call("gc_fused_load", s.h, *[_ptr(t) for t in state["start"][state["passes"] % 2]], 1)
    state["passes"] += 1
    s.step(case["steps"], 1)
    _lib.call("gc_fused_store", s.h, _ptr(state["pos"]), _ptr(state["vel"]), _ptr(state["rho"]), _ptr(state["press"]),
              _ptr(state["force"]), _ptr(None), _ptr(state["nthro"]), 1)
    cells = state["cells"]
    if cells:
        _lib.call("gc_fused_store_cells", s.h, *[_ptr(cells[k]) for k in _CELLS], 1)
    return dict(pos=state["pos"] + state["nthro"] * state["lengths"], vel=state["vel"], rho=state["rho"],
                press=state["press"], force=state["force"], **_membrane(case, cells))


def work(case):
    """Each step reads position, velocity and force of every particle and
    writes them, reads every triangle (16 B) and edge (32 B) record, and
    evaluates every pair within the cut-off from both ends: about 4/3 pi 27
    partners, 20 operations for the density and 70 for the force."""
    cfgs = _configs(case)
    n, ntri, nedge = sum(c.n for c in cfgs), sum(c.ntri for c in cfgs), sum(c.nedge for c in cfgs)
    return {"bytes": case["steps"] * (72.0 * n + 16.0 * ntri + 32.0 * nedge) + 44.0 * n,
            "flops": case["steps"] * n * 113.0 * 90.0}


# ---------------------------------------------------------------------------
# The method in 64 bits
# ---------------------------------------------------------------------------
def _mix64(z):
    m = (1 << 64) - 1
    z = (z + 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def _pair_noise(i, j, key):
    """Three variates of the pair (i, j), antisymmetric (Philox2x32-10)."""
    c0, c1, low = torch.minimum(i, j), torch.maximum(i, j), 0xFFFFFFFF
    for _ in range(10):
        p = c0 * 0xD256D193
        c0, c1 = (p >> 32 & low) ^ key ^ c1, p & low
        key = (key + 0x9E3779B9) & low
    u = torch.stack([c0 & 0x1FFFFF, c0 >> 21 | (c1 & 0x3FF) << 11, c1 >> 10 & 0x1FFFFF], 1)
    return torch.where(i < j, 1.0, -1.0)[:, None] * (math.sqrt(12.0) * ((u.double() + 0.5) / 2097152.0 - 0.5))


class _Model:
    def __init__(self, cfg, vel, noise):
        self.c, self.ph, self.noise = cfg, cfg.phys, noise
        f64 = lambda a: torch.as_tensor(np.asarray(a), device=DEVICE).double()
        idx = lambda a: torch.as_tensor(np.asarray(a), device=DEVICE).long()
        self.f64 = f64
        self.x, self.v, self.vh = f64(cfg.coor), f64(vel), f64(cfg.velhalf)
        self.f = torch.zeros_like(self.x)
        b = cfg.bbox.astype(np.float32)
        self.lo, self.L = f64(b[0::2]), f64(b[1::2] - b[0::2])
        self.periodic = torch.tensor([bool(cfg.pmask >> a & 1) for a in range(3)], device=DEVICE)
        n = cfg.n
        ids = torch.arange(n, device=DEVICE)
        self.b1, self.b2 = ids < cfg.n_b1, (ids >= cfg.n_b1) & (ids < cfg.n_b1 + cfg.n_b2)
        self.mobile, self.memb = ids >= cfg.n_b1 + cfg.n_b2, ids >= cfg.n_cell_start
        self.rho0 = float(np.float32(cfg.den_init))
        self.rho = torch.full((n,), self.rho0, dtype=torch.float64, device=DEVICE)
        self.k = -1
        f32 = lambda x: float(np.float32(x))
        for name in ("sound1", "sound2", "shear_vis", "bulk_vis", "temp", "dt", "mass", "vvsigma", "sur_energy", "max_cut",
                     "zero_len", "sca_fac"):
            setattr(self, name, f32(getattr(cfg.phys, name)))
        self.gx = f32(cfg.phys.ext_force * cfg.phys.mass)
        if cfg.ncell:
            self.tri, self.edge = idx(cfg.tri) - 1, idx(cfg.edge)[:, :4] - 1
            self.cell = idx(cfg.celltab)
            self.tcell = torch.repeat_interleave(torch.arange(cfg.ncell, device=DEVICE), idx(cfg.betri)[:, 1] - idx(cfg.betri)[:, 0] + 1)
            self.first = self.tri[idx(cfg.betri)[:, 0], 0]
            self.mod = [f64(a) for a in cfg.edge_params()]
            self.reference()

    # -- pairs within `cut` among the particles `which` ---------------------
    def pairs(self, x, cut, which=None):
        x = x if which is None else x[which]
        w = torch.where(self.periodic, self.lo + torch.remainder(x - self.lo, self.L), x)
        lo = torch.where(self.periodic, self.lo, w.min(0).values - 1e-6)
        L = torch.where(self.periodic, self.L, w.max(0).values + 1e-6 - lo)
        nc = torch.clamp((L / (cut * 1.0001)).floor().long(), min=1)
        per = self.periodic.tolist()
        c = torch.minimum(((w - lo) / L * nc).floor().long(), nc - 1).clamp(min=0)
        key = c[:, 0] + nc[0] * (c[:, 1] + nc[1] * c[:, 2])
        order = torch.argsort(key)
        total = int(nc.prod())
        start = torch.zeros(total + 1, dtype=torch.long, device=DEVICE)
        start[1:] = torch.bincount(key, minlength=total).cumsum(0)
        for off in range(27):
            d = [off % 3 - 1, off // 3 % 3 - 1, off // 9 - 1]
            ok, q = torch.ones(x.shape[0], dtype=torch.bool, device=DEVICE), []
            for a in range(3):
                t = c[:, a] + d[a]
                if per[a]:
                    t = t % nc[a]
                else:
                    ok &= (t >= 0) & (t < nc[a])
                    t = t.clamp(min=0).minimum(nc[a] - 1)
                q.append(t)
            kk = q[0] + nc[0] * (q[1] + nc[1] * q[2])
            cnt = torch.where(ok, start[kk + 1] - start[kk], 0)
            i = torch.repeat_interleave(torch.arange(x.shape[0], device=DEVICE), cnt)
            at = torch.arange(i.numel(), device=DEVICE) - (cnt.cumsum(0) - cnt)[i]
            j = order[start[kk][i] + at]
            r2 = self.image(w[i] - w[j]).square().sum(1)
            keep = (r2 < cut * cut) & (i != j)
            yield i[keep], j[keep]

    def image(self, d):
        return torch.where(self.periodic, d - self.L * torch.round(d / self.L), d)

    def delta(self, i, j):
        d = self.image(self.x[i] - self.x[j])
        return d, d.square().sum(1).sqrt()

    # -- membranes ----------------------------------------------------------
    def geometry(self):
        m = self.x[self.c.n_cell_start:]
        self.m = m
        p1, p2, p3 = (m[self.tri[:, q]] for q in range(3))
        xi = torch.linalg.cross(p2 - p1, p3 - p1)
        len_ = xi.square().sum(1).sqrt()
        self.xi, self.tarea, self.tnorm, self.tcen = xi, 0.5 * len_, xi / len_[:, None], (p1 + p2 + p3) / 3.0
        o = m[self.first][self.tcell]
        vol = ((p1 - o) * torch.linalg.cross(p2 - o, p3 - o)).sum(1) / 6.0
        add = lambda v: torch.zeros(self.c.ncell, dtype=torch.float64, device=DEVICE).index_add_(0, self.tcell, v)
        self.area, self.vol = add(self.tarea), add(vol)
        self.parea = torch.zeros(self.c.ncp, dtype=torch.float64, device=DEVICE)
        for q in range(3):
            self.parea.index_add_(0, self.tri[:, q], self.tarea / 3.0)

    def edges(self):
        e = [self.m[self.edge[:, q]] for q in range(4)]
        return e[1] - e[0], e[2] - e[0], e[3] - e[0]

    @staticmethod
    def dihedral(xi, xk, xl):
        """Angle of (i, j, k, l) with j at the origin, and its gradients."""
        dot = lambda a, b: (a * b).sum(1, keepdim=True)
        rij, rkj, rkl = xi, xk, xk - xl
        m, n = torch.linalg.cross(rij, rkj), torch.linalg.cross(rkj, rkl)
        m2, n2, kj = dot(m, m), dot(n, n), dot(rkj, rkj).sqrt()
        phi = torch.atan2(dot(m, rkl) * kj, dot(m, n))
        gi, gl = kj / m2 * m, -kj / n2 * n
        a, b = dot(rij, rkj) / kj ** 2, dot(rkl, rkj) / kj ** 2
        return phi, gi, (a - 1.0) * gi - b * gl, (b - 1.0) * gl - a * gi, gl

    def reference(self):
        self.geometry()
        b, c, d = self.edges()
        self.l0 = b.square().sum(1).sqrt()
        x0, u = 1.0 / 2.2, 1.0 - 1.0 / 2.2
        kwlc, kmod = 0.25 / u ** 2 - 0.25 + x0, x0 / (2.0 * u ** 3) - 0.25 / u ** 2 + 0.25
        self.ktp = self.mod[0] * 4.0 * self.l0 / (math.sqrt(3.0) * (kmod + 3.0 * kwlc))   # kT / p
        self.hpow = self.ktp * self.l0 ** 2 * kwlc
        self.kb = 2.0 * self.mod[1] / math.sqrt(3.0)
        self.phi0 = self.dihedral(c, b, d)[0]
        self.reftarea, self.refarea, self.refvol = self.tarea, self.area, self.vol

    def membranes(self):
        self.geometry()
        F = torch.zeros_like(self.m)
        b, c, d = self.edges()
        r = b.square().sum(1).sqrt()
        x = r / (2.2 * self.l0)
        fm = -self.ktp * (0.25 / (1.0 - x) ** 2 - 0.25 + x) + self.hpow / r ** 2
        s = -(fm / r)[:, None] * b
        phi, gi, gj, gk, gl = self.dihedral(c, b, d)
        dE = self.kb[:, None] * torch.sin(phi - self.phi0)
        for q, f in ((0, s - dE * gj), (1, -s - dE * gk), (2, -dE * gi), (3, -dE * gl)):
            F.index_add_(0, self.edge[:, q], f)
        p1, p2, p3 = (self.m[self.tri[:, q]] for q in range(3))
        hl, hg, hv = self.mod[2:]
        cA = hg * ((self.area - self.refarea) / self.refarea)[self.tcell] + hl * (self.tarea - self.reftarea) / self.reftarea
        cV = hv * ((self.vol - self.refvol) / self.refvol)[self.tcell] / 6.0
        for q, e in ((0, p3 - p2), (1, p1 - p3), (2, p2 - p1)):
            F.index_add_(0, self.tri[:, q], -cV[:, None] * self.xi - cA[:, None] * 0.5 * torch.linalg.cross(self.tnorm, e))
        self.defforce, self.aggforce = F, torch.zeros_like(F)
        if self.sur_energy and self.max_cut:
            for i, j in self.pairs(self.x, self.max_cut, self.memb):
                other = self.cell[i] != self.cell[j]
                i, j = i[other], j[other]
                d = self.image(self.m[i] - self.m[j])
                r = d.square().sum(1).sqrt()
                ex = torch.exp(self.sca_fac * (self.zero_len - r))
                f = self.sur_energy * self.sca_fac * (ex * ex - ex) * (self.parea[i] + self.parea[j]) / r
                self.aggforce.index_add_(0, i, f[:, None] * d)

    # -- one step -------------------------------------------------------------
    def walls(self):
        if not self.c.n_b2:
            return
        num, den = torch.zeros_like(self.x), torch.zeros_like(self.rho)
        for i, j in self.wall_pairs:
            r = self.delta(i, j)[1]
            w = (1.0 - r) ** 4 * (1.0 + 4.0 * r)
            num.index_add_(0, i, w[:, None] * self.v[j])
            den.index_add_(0, i, w)
        mean = torch.where(den[:, None] > 0, num / den.clamp(min=1e-300)[:, None], self.vh)
        self.v = torch.where(self.b2[:, None], 2.0 * self.vh - mean, self.v)

    def step(self):
        self.k += 1
        dt, m, mob = self.dt, self.mass, self.mobile[:, None]
        self.x = torch.where(mob, self.x + dt * self.v + 0.5 * dt * dt / m * self.f, self.x)
        found = list(self.pairs(self.x, 1.0))
        self.vh = torch.where(mob, self.v + 0.5 * dt / m * self.f, self.vh)
        self.v = torch.where(mob, self.v + self.vvsigma * dt / m * self.f, self.v)
        wnorm, fnorm = 21.0 / (2.0 * math.pi), 210.0 / math.pi
        total = torch.ones_like(self.rho)
        self.wall_pairs = []
        for i, j in found:
            r = self.delta(i, j)[1]
            total.index_add_(0, i, torch.where(self.b1[j], 0.0, (1.0 - r) ** 4 * (1.0 + 4.0 * r)))
            w = self.b2[i] & self.mobile[j]
            self.wall_pairs.append((i[w], j[w]))
        self.rho = torch.where(self.mobile, m * wnorm * total, self.rho)
        self.walls()
        c2 = torch.where(self.memb, self.sound2 ** 2, self.sound1 ** 2)
        self.press = torch.where(self.b1, 0.0, c2 * (self.rho - self.rho0))
        den = self.rho / m
        A, B = 5.0 * self.shear_vis / 3.0 - self.bulk_vis, 5.0 * (self.bulk_vis + self.shear_vis / 3.0)
        amp = 2.0 * self.temp / dt if self.noise else 0.0
        key = _mix64((self.ph.seed * 0x9E3779B97F4A7C15 + self.k) & ((1 << 64) - 1)) >> 32
        self.f = torch.zeros_like(self.x)
        for i, j in found:
            w = self.mobile[i]
            i, j = i[w], j[w]
            d, r = self.delta(i, j)
            if self.c.n_b1:
                rep = self.b1[j] & (r < 1.0 / 3.0)
                q2 = 1.0 / (9.0 * r[rep] ** 2)
                self.f.index_add_(0, i[rep], (self.sound1 ** 2 * (q2 ** 6 - q2 ** 2) * 9.0 * q2)[:, None] * d[rep])
                w = ~self.b1[j]
                i, j, d, r = i[w], j[w], d[w], r[w]
            e, F = d / r[:, None], fnorm * (1.0 - r) ** 3
            vij = self.v[i] - self.v[j]
            fdd = F / (den[i] * den[j])
            pair = ((self.press[i] / den[i] ** 2 + self.press[j] / den[j] ** 2) * F)[:, None] * d
            pair -= fdd[:, None] * (A * vij + B * (e * vij).sum(1, keepdim=True) * e)
            if amp:
                xi = _pair_noise(i, j, key)
                pair += (amp * fdd).clamp(min=0.0).sqrt()[:, None] * (
                    math.sqrt(A) * xi + (math.sqrt(A + B) - math.sqrt(A)) * (e * xi).sum(1, keepdim=True) * e)
            self.f.index_add_(0, i, pair)
        self.f[:, 0] += torch.where(self.mobile, self.gx, 0.0)
        if self.c.ncell:
            self.membranes()
            self.f[self.c.n_cell_start:] += self.defforce + self.aggforce
        self.v = torch.where(mob, self.vh + 0.5 * dt / m * self.f, self.v)
        self.walls()


def exact(case, seed):
    models = []
    for cfg, vel in _inputs(case, seed):
        m = _Model(cfg, vel, case["noise"])
        for _ in range(case["steps"]):
            m.step()
        models.append(m)
    cat = lambda f: torch.cat([f(m) for m in models])
    out = dict(pos=cat(lambda m: m.x), vel=cat(lambda m: m.v), rho=cat(lambda m: m.rho), press=cat(lambda m: m.press),
               force=cat(lambda m: m.f))
    if case["api"] == "dropin" and not models[0].c.ncell:
        m = models[0]
        out["pos"] = torch.where(m.periodic & m.mobile[:, None], m.lo + torch.remainder(m.x - m.lo, m.L), m.x)
    models = [m for m in models if m.c.ncell]
    if models:
        out.update(_membrane(case, dict(
            area=cat(lambda m: m.area), vol=cat(lambda m: m.vol), defforce=cat(lambda m: m.defforce),
            aggforce=cat(lambda m: m.aggforce), trinordir=cat(lambda m: m.tnorm), tricenter=cat(lambda m: m.tcen),
            pararea=cat(lambda m: m.parea))))
    return out
