"""The measured workloads: what a program has the engines do, through their public calls.

Every case is one *pass* of a stepping program:

* ``gas`` / ``bed`` / ``sheet`` -- :class:`HM2D`: the settling disc gas (dilute), a
  settled bed of touching discs (three contacts per disc, walls and friction
  at work) and the bonded ice sheet under a rigid indenter. ``solve`` cases
  upload a state, run it and read it back (one request of a parameter study);
  the others advance a live engine by a block of steps and read the state, as
  a monitored run does.
* ``batch`` -- :class:`Batch`: the mixed ensemble (bonded-ice indentations and
  column collapses, counts log-uniform) advanced by one step block, then the
  ledgers of all runs and the state of two.
* ``ice2d`` -- :class:`IceDEM`: the 21 x 5 icebreaking demonstration (and other
  lattice sizes), from a seeded state.
* ``ice3d`` -- :class:`IceDEM3D`: the 3-D indentation specimens.

Bytes and operations of a pass count one reading and one writing of every
disc's state per step, its list head, and the bond and history data that the
step's laws cannot do without.
"""

from __future__ import annotations

import math
from dataclasses import replace

import numpy as np
import torch

from tensordem_gb300.batch import Batch, BatchConfig, ensemble_case
from tensordem_gb300.dem import DEMConfig, IceDEM
from tensordem_gb300.dem3d import DEM3DConfig, IceDEM3D
from tensordem_gb300.hm2d import HM2D, HM2DConfig, granular_gas_case, ice_sheet_case, rayleigh_dt

_DEV = "cuda"


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _gas(n_side, steps, *, precision=32, solve=False, variant=-1):
    return dict(kind="gas", nx=n_side, ny=n_side, steps=steps, precision=precision, solve=solve, variant=variant)


def _bed(nx, ny, steps, *, precision=32, solve=False, variant=-1):
    return dict(kind="bed", nx=nx, ny=ny, steps=steps, precision=precision, solve=solve, variant=variant)


def _sheet(nx, ny, steps, *, precision=32, solve=False, variant=-1):
    return dict(kind="sheet", nx=nx, ny=ny, steps=steps, precision=precision, solve=solve, variant=variant)


def _batch(runs, n_min, n_max, steps, *, precision=32):
    return dict(kind="batch", runs=runs, n_min=n_min, n_max=n_max, steps=steps, precision=precision)


def listed() -> list[dict]:
    return [
        # a small granular run, uploaded, stepped and read back: latency of the step loop
        dict(_bed(20, 15, 100, solve=True), name="bed_300_solve"),
        # a few thousand dilute discs, odd count
        dict(_gas(57, 200, solve=True), name="gas_3k_solve"),
        # a settled bed of 50,071 touching discs, monitored every 100 steps
        dict(_bed(311, 161, 100), name="bed_50k"),
        # the 1,048,576-disc settling run, with the step shape that the timed bench picks
        dict(_gas(1024, 100, variant=10), name="gas_1m"),
        # four million discs: the state exceeds the L2 cache
        dict(_gas(2048, 40), name="gas_4m"),
        # the plain FP64 form on a bed, which the FP32 results are checked against
        dict(_bed(257, 255, 50, precision=64), name="bed_65k_fp64"),
        # a small bonded sheet, uploaded with its bonds, indented and read back
        dict(_sheet(97, 24, 200, solve=True), name="sheet_2k_solve"),
        # the 1,048,576-disc bonded sheet, with the step shape that autotuning picks
        dict(_sheet(2048, 512, 40, variant=11), name="sheet_1m"),
        # a light serving load: 32 small mixed runs
        dict(_batch(32, 100, 2000, 100), name="batch_32"),
        # 256 mixed runs of 100 to 20,000 discs
        dict(_batch(256, 100, 20000, 40), name="batch_256"),
        # the 21 x 5 demonstration: 250 steps of the FP64 reference mode
        dict(kind="ice2d", nx=21, ny=5, steps=250, name="ice2d_demo"),
        # an 8,000-particle 3-D indentation specimen
        dict(kind="ice3d", nx=40, ny=20, nz=10, steps=20, name="ice3d_8k"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["gas", "bed", "gas", "bed", "sheet", "sheet", "batch", "batch", "fp64", "ice2d", "ice3d"])
    if kind == "gas":
        side = _log_int(rng, 9, 2000)
        solve = side * side < 20000
        return _gas(side, _log_int(rng, 30, 120) if side < 1100 else _log_int(rng, 15, 40), solve=solve,
                    variant=rng.choice([-1, -1, 10]))
    if kind == "bed":
        n = _log_int(rng, 100, 600_000)
        nx = max(4, int(math.sqrt(n * rng.uniform(0.5, 3.0))))
        return _bed(nx, max(4, n // nx), _log_int(rng, 30, 120), solve=n < 20000)
    if kind == "fp64":
        n = _log_int(rng, 100, 200_000)
        nx = max(4, int(math.sqrt(n * rng.uniform(0.5, 3.0))))
        if rng.random() < 0.5:
            return _bed(nx, max(4, n // nx), _log_int(rng, 20, 60), precision=64, solve=n < 20000)
        return _sheet(2 * nx, max(6, n // (2 * nx)), _log_int(rng, 20, 60), precision=64, solve=n < 20000)
    if kind == "sheet":
        n = _log_int(rng, 300, 600_000)
        nx = max(24, int(math.sqrt(4.0 * n)))
        return _sheet(nx, max(6, n // nx), _log_int(rng, 30, 120) if n < 100_000 else 40, solve=n < 20000,
                      variant=rng.choice([-1, 11]))
    if kind == "batch":
        runs, n_max = _log_int(rng, 5, 200), _log_int(rng, 400, 20000)
        return _batch(runs, 100, n_max, 30 if runs * n_max > 10**6 else _log_int(rng, 30, 100),
                      precision=rng.choice([32, 32, 32, 64]) if runs < 30 else 32)
    if kind == "ice2d":
        return dict(kind="ice2d", nx=rng.randrange(5, 36), ny=rng.randrange(3, 13), steps=_log_int(rng, 60, 250))
    nx, ny, nz = rng.choice([(9, 5, 3), (20, 10, 6), (13, 7, 5), (31, 11, 9)])
    return dict(kind="ice3d", nx=nx, ny=ny, nz=nz, steps=_log_int(rng, 15, 60))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _bed_case(case, seed):
    """A settled bed: hexagonal rows of nearly equal discs (radii r0 (1 +- 2e-4)) whose
    neighbours overlap or miss by up to 2e-4 of a diameter, between side walls and on a floor,
    with the residual motion of a settled bed."""
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    n = nx * ny
    r0, density, young, poisson, skin = 1e-3, 2500.0, 5e9, 0.25, 0.1e-3
    radius = r0 * (1.0 + rng.uniform(-2e-4, 2e-4, n))
    width = (2 * nx + 1) * r0
    ncx = max(1, int(width / (2.0 * r0 * (1 + 2e-4) + skin)))
    cell = float(np.float32(width / ncx)) if case["precision"] == 32 else width / ncx
    ncy = int(math.ceil(((ny - 1) * math.sqrt(3.0) * r0 + 6.0 * r0) / cell))
    jj, ii = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    pos = np.stack(((2 * ii + jj % 2 + 1).ravel() * r0, (1 + jj * math.sqrt(3.0)).ravel() * r0), axis=1)
    mass = density * math.pi * radius**2 * (2.0 * radius)
    cfg = HM2DConfig(n=n, ncx=ncx, ncy=ncy, cell=cell, skin=skin, dt=0.2 * rayleigh_dt(0.999 * r0, density, young, poisson),
                     young=young, poisson=poisson, restitution=0.8, mu=0.5, mu_wall=0.5, precision=case["precision"])
    state = dict(pos=pos, vel=rng.normal(0.0, 0.01, (n, 2)), omega=rng.normal(0.0, 5.0, n), radius=radius, mass=mass,
                 inertia=0.5 * mass * radius**2)
    return cfg, state, None, None


def _hm_case(case, seed):
    """(config, state, bonds, strength) of an HM2D case, host FP64."""
    if case["kind"] == "gas":
        cfg, state = granular_gas_case(case["nx"], seed=seed, precision=case["precision"])
        state["omega"] = np.random.default_rng(seed + 1).normal(0.0, 50.0, cfg.n)
        return cfg, state, None, None
    if case["kind"] == "bed":
        return _bed_case(case, seed)
    # a request's indenter moves at 5 m/s, a monitored run's at 0.5 m/s; it already touches the
    # top row, and the sheet carries the waves of the impact as residual motion of its discs.
    # Walls keep fragments in the tank; small sheets take a smaller indenter.
    big = case["nx"] >= 1000
    cfg, state, bonds, strength = ice_sheet_case(case["nx"], case["ny"], seed=seed, precision=case["precision"],
                                                 indenter_speed=5.0 if case["solve"] else 0.5,
                                                 indenter_radius=2.0 if big else 0.3, steps=20000, max_neighbors=12)
    state["vel"] = _residual(state, seed)
    cx, cy = cfg.indenter_center
    cfg = replace(cfg, indenter_center=(cx, cy - 0.03 * 0.05), walls=15)
    return cfg, state, bonds, strength


def _residual(state, seed):
    """Velocities of a sheet under load: the waves of the impact, clamped discs at rest."""
    vel = np.random.default_rng(seed + 1).normal(0.0, 0.05, state["pos"].shape)
    vel[~np.isfinite(state["mass"])] = 0.0
    return vel


def _upload(state):
    s = state
    s["engine"].set_state(*s["inputs"])
    if s["bonds"] is not None:
        s["engine"].set_bonds(s["bonds"], s["strength"])


def _batch_instances(case, seed):
    # the runs' sizes and materials are the case's, their states the seed's; the indentations are
    # under way: the indenter touches the strip and descends at 0.1 m/s
    specs = ensemble_case(case["runs"], seed=0, n_min=case["n_min"], n_max=case["n_max"], steps=20000)
    got = []
    for s, k in zip(specs, np.random.default_rng(seed).integers(0, 2**62, len(specs))):
        i = replace(s, seed=int(k)).build()
        if s.kind == "ice":
            i.state["vel"] = _residual(i.state, int(k))
            cx, cy = i.config.indenter_center
            i.config = replace(i.config, indenter_center=(cx, cy - 0.05 * 0.05), indenter_velocity=(0.0, -0.1))
        got.append(i)
    return got


def _ice2d_velocities(case, seed, n):
    return torch.from_numpy(np.random.default_rng(seed).normal(0.0, 0.02, (n, 2))).to(_DEV)


def _ice3d_config(case):
    return DEM3DConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"], breaking_strain=0.004,
                       shear_breaking_strain=0.008, friction_coefficient=0.3, restitution_coefficient=0.7)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("gas", "bed", "sheet"):
        cfg, st, bonds, strength = _hm_case(case, seed)
        eng = HM2D(cfg)
        if case["variant"] >= 0:
            eng.variant = case["variant"]
        inputs = [torch.from_numpy(np.ascontiguousarray(st[k])).to(_DEV)
                  for k in ("pos", "vel", "omega", "radius", "mass", "inertia")]
        state = dict(kind=kind, engine=eng, inputs=inputs, bonds=bonds, strength=strength, steps=case["steps"],
                     solve=case["solve"])
        _upload(state)
        eng.step(0)  # builds the step graph ahead, as the command line does
        return state
    if kind == "batch":
        insts = _batch_instances(case, seed)
        b = Batch(BatchConfig(particle_capacity=sum(i.n for i in insts) + 64,
                              key_capacity=sum(i.keys for i in insts) + 64, max_instances=max(64, len(insts)),
                              precision=case["precision"]))
        ids = [b.admit(i) for i in insts]
        b.step(0)
        return dict(kind=kind, batch=b, ids=ids, steps=case["steps"])
    if kind == "ice2d":
        sim = IceDEM(DEMConfig(nx=case["nx"], ny=case["ny"], breaking_strain=0.01, shear_breaking_strain=0.02))
        first = dict(positions=sim.positions.clone(),
                     velocities=_ice2d_velocities(case, seed, len(sim.positions)), alive=sim.alive.clone())
        first["velocities"][sim.fixed] = 0.0
        return dict(kind=kind, sim=sim, first=first, steps=case["steps"])
    sim = IceDEM3D(_ice3d_config(case))
    sim.velocities = _ice3d_velocities(seed, sim)
    return dict(kind=kind, sim=sim, steps=case["steps"])


def _ice3d_velocities(seed, sim):
    v = torch.from_numpy(np.random.default_rng(seed).normal(0.0, 0.01, tuple(sim.positions.shape))).to(_DEV)
    v[sim.fixed] = 0.0
    return v


_LEDGER = ("kinetic", "potential", "hertz", "tangential", "dissipated", "bond_elastic", "fracture_released",
           "tool_work", "broken", "peak_load", "reaction_x", "reaction_y")


def run(state):
    kind = state["kind"]
    if kind in ("gas", "bed", "sheet"):
        if state["solve"]:
            _upload(state)
        state["engine"].step(state["steps"])
        return state["engine"].state()
    if kind == "batch":
        b, ids = state["batch"], state["ids"]
        b.step(state["steps"])
        led = b.ledgers(ids)
        out = {k: np.array([row[k] for row in led]) for k in _LEDGER}
        for at in (0, -1):
            one = b.read(ids[at])
            out.update({f"{k}_{at}": one[k] for k in ("pos", "vel", "omega", "force", "torque")})
        return out
    sim = state["sim"]
    if kind == "ice2d":
        # the demonstration again from its first state
        sim.positions.copy_(state["first"]["positions"])
        sim.velocities.copy_(state["first"]["velocities"])
        sim.alive.copy_(state["first"]["alive"])
        sim.failure_mode.zero_()
        sim.failure_time_s.fill_(-1.0)
        sim.failure_extension_m.zero_()
        sim.failure_energy_J.zero_()
        sim.time, sim.step_count = 0.0, 0
        sim.run(state["steps"])
        force, reaction = sim.forces()
        return dict(positions=sim.positions, velocities=sim.velocities, force=force, reaction=reaction,
                    alive=sim.alive, failure_mode=sim.failure_mode, failure_time=sim.failure_time_s)
    sim.run(state["steps"])
    return dict(positions=sim.positions, velocities=sim.velocities, alive=sim.alive,
                failure_mode=sim.failure_mode, reaction=sim.last_reaction)


def work(case):
    kind, steps = case["kind"], case["steps"]
    if kind in ("gas", "bed", "sheet", "batch"):
        word = case["precision"] // 8
        if kind == "batch":
            n = case["runs"] * (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
            bonds, touching = 0.5 * 2.8 * n, 0.0
        else:
            n = case["nx"] * case["ny"]
            bonds = 3.0 * n if kind == "sheet" else 0.0
            touching = 3.0 * n if kind == "bed" else 0.0
        # position, velocity and remainder read and written, the list head read; per contact
        # side its history read and written; per bond side its partner, reference vector,
        # strength and shear displacement read, the displacement written
        disc = 2 * (8 * word + (8 if word == 4 else 0)) + 16
        per_step = n * disc + touching * 4 * word + 2 * bonds * (4 + 7 * word)
        return {"bytes": steps * per_step, "flops": steps * (40.0 * n + 60.0 * touching + 2 * 90.0 * bonds)}
    n = case["nx"] * case["ny"] * case.get("nz", 1)
    if kind == "ice2d":
        return {"bytes": steps * n * 64.0, "flops": steps * n * (3.4 * 2 * 60.0 + 60.0)}
    return {"bytes": steps * n * 96.0, "flops": steps * n * (12.0 * 2 * 90.0 + 200.0)}


# ---------------------------------------------------------------------------
# The same passes in plain torch FP64
# ---------------------------------------------------------------------------
def _pinv2(cov):
    """Pseudo-inverses of symmetric positive semi-definite 2 x 2 matrices given as rows of four."""
    det = cov[:, 0] * cov[:, 3] - cov[:, 1] * cov[:, 2]
    trace = cov[:, 0] + cov[:, 3]
    full = det > 1e-10 * trace**2
    inv = torch.stack((cov[:, 3], -cov[:, 1], -cov[:, 2], cov[:, 0]), 1) / torch.where(full, det, torch.ones_like(det))[:, None]
    one = cov / torch.where(trace > 0, trace**2, torch.ones_like(trace))[:, None]
    return torch.where(full[:, None], inv, one).reshape(-1, 2, 2)


class _Discs:
    """Hertz-Mindlin discs, bonds and indenters of several independent runs at once, velocity-Verlet, FP64."""

    def __init__(self, runs):
        """runs: (config, state, bonds, strength) each."""
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_DEV)  # noqa: E731
        counts = [r[0].n for r in runs]
        self.first = np.concatenate(([0], np.cumsum(counts)))
        self.n = int(self.first[-1])
        cat = lambda k: t(np.concatenate([r[1][k] for r in runs]))  # noqa: E731
        self.x, self.v, self.w, self.r = cat("pos"), cat("vel"), cat("omega"), cat("radius")
        mass = cat("mass")
        self.m = torch.where(torch.isfinite(mass), mass, torch.zeros_like(mass))
        self.im = torch.where(torch.isfinite(mass), 1.0 / mass, torch.zeros_like(mass))
        inertia = cat("inertia")
        self.ii = torch.where(torch.isfinite(inertia), 1.0 / inertia, torch.zeros_like(inertia))
        self.inst = torch.repeat_interleave(torch.arange(len(runs), device=_DEV), torch.tensor(counts, device=_DEV))
        cfgs = [r[0] for r in runs]
        per = lambda f: t([f(c) for c in cfgs])[self.inst]  # noqa: E731

        def beta(c):
            return 0.0 if c.restitution >= 1 else -math.log(c.restitution) / math.hypot(math.log(c.restitution), math.pi)

        self.e2 = per(lambda c: c.young / (1.0 - c.poisson**2))
        self.g8 = per(lambda c: 2.0 * c.young / ((2.0 - c.poisson) * (1.0 + c.poisson)))
        self.damp = per(lambda c: 2.0 * math.sqrt(5.0 / 6.0) * beta(c))
        self.mu, self.muw = per(lambda c: c.mu), per(lambda c: c.mu_wall)
        self.dt = per(lambda c: c.dt)
        self.skin = per(lambda c: c.skin)
        self.cell = per(lambda c: c.cell)
        self.g = torch.stack((per(lambda c: c.gravity[0]), per(lambda c: c.gravity[1])), 1)
        self.box = torch.stack((per(lambda c: c.box[0]), per(lambda c: c.box[1])), 1)
        self.walls = torch.tensor([c.walls for c in cfgs], device=_DEV)[self.inst]
        self.stride = torch.tensor([c.ncx + 4 for c in cfgs], device=_DEV)[self.inst]
        cells = np.array([(c.ncx + 4) * (c.ncy + 4) for c in cfgs])
        self.base = torch.from_numpy(np.concatenate(([0], np.cumsum(cells)))[:-1]).to(_DEV)[self.inst]
        self.nkeys = int(cells.sum())
        self.wall_xi = torch.zeros((4, self.n, 2), dtype=torch.float64, device=_DEV)
        self.keys = torch.zeros(0, dtype=torch.int64, device=_DEV)
        self.xi = torch.zeros((0, 2), dtype=torch.float64, device=_DEV)
        self.evals = 0
        # bonds
        pairs = [np.sort(np.asarray(r[2], dtype=np.int64), axis=1) + self.first[k] for k, r in enumerate(runs)
                 if r[2] is not None and len(r[2])]
        self.nb = sum(len(p) for p in pairs)
        if self.nb:
            b = torch.from_numpy(np.concatenate(pairs)).to(_DEV)
            self.bi, self.bj = b[:, 0].contiguous(), b[:, 1].contiguous()
            self.bf = t(np.concatenate([r[3] for r in runs if r[2] is not None and len(r[2])]))
            self.bref = self.x[self.bj] - self.x[self.bi]
            self.bl0 = self.bref.square().sum(1).sqrt()
            self.kn, self.ks = per(lambda c: c.bond_kn)[self.bi], per(lambda c: c.bond_ks)[self.bi]
            self.zeta = per(lambda c: c.bond_damping)[self.bi]
            self.et, self.es = per(lambda c: c.breaking_strain)[self.bi], per(lambda c: c.shear_breaking_strain)[self.bi]
            self.alive = torch.ones(self.nb, dtype=torch.bool, device=_DEV)
            self.us = torch.zeros((self.nb, 2), dtype=torch.float64, device=_DEV)
            outer = (self.bref[:, :, None] * self.bref[:, None, :]).reshape(-1, 4)
            cov = torch.zeros((self.n, 4), dtype=torch.float64, device=_DEV)
            cov.index_add_(0, self.bi, outer).index_add_(0, self.bj, outer)
            self.pinv = _pinv2(cov)
        self.irad = per(lambda c: c.indenter_radius)
        self.icen = torch.stack((per(lambda c: c.indenter_center[0]), per(lambda c: c.indenter_center[1])), 1)
        self.ivel = torch.stack((per(lambda c: c.indenter_velocity[0]), per(lambda c: c.indenter_velocity[1])), 1)
        self.has_ind = any(c.indenter_radius > 0 for c in cfgs)
        self.sums = lambda per_disc: torch.zeros(len(runs), dtype=torch.float64, device=_DEV).index_add_(  # noqa: E731
            0, self.inst, per_disc)
        self.dissipated = torch.zeros(len(runs), dtype=torch.float64, device=_DEV)
        self.pi = None

    def candidates(self):
        """Every pair i < j within r_i + r_j + skin, by cells of the runs' grids."""
        c = torch.floor(self.x / self.cell[:, None]).to(torch.int64) + 2
        key = self.base + c[:, 1] * self.stride + c[:, 0]
        order = torch.argsort(key, stable=True)
        start = torch.searchsorted(key[order], torch.arange(self.nkeys + 1, device=_DEV))
        ids = torch.arange(self.n, device=_DEV)
        got = []
        most = int((start[1:] - start[:-1]).max())
        for dy, dx in ((0, 0), (0, 1), (1, -1), (1, 0), (1, 1)):
            k = torch.clamp(key + dy * self.stride + dx, 0, self.nkeys - 1)
            lo, num = start[k], start[k + 1] - start[k]
            for s in range(most):
                a = ids[num > s]
                b = order[lo[a] + s]
                if dx == 0 and dy == 0:
                    keep = a < b
                    a, b = a[keep], b[keep]
                near = ((self.x[b] - self.x[a]).square().sum(1).sqrt() <= self.r[a] + self.r[b] + self.skin[a]) & \
                    (self.inst[a] == self.inst[b])
                got.append(torch.stack((torch.minimum(a, b)[near], torch.maximum(a, b)[near]), 1))
        p = torch.cat(got)
        pkey = torch.sort(p[:, 0] * self.n + p[:, 1]).values
        self.pi, self.pj = pkey // self.n, pkey % self.n

    def contact(self, delta, nrm, reff, meff, lever, vrel, xi, e2, g8, damp, mu, dt):
        """Force along -normal and tangent, new history, dissipation and elastic energy of touching contacts."""
        sq = (reff * delta).sqrt()
        sn = e2 * sq
        fel = (2.0 / 3.0) * sn * delta
        vn = (vrel * nrm).sum(1)
        fn = torch.clamp(fel + damp * (sn * meff).sqrt() * vn, min=0.0)
        vt = vrel - vn[:, None] * nrm
        xi = xi + vt * dt[:, None]
        xi = xi - (xi * nrm).sum(1)[:, None] * nrm
        st = g8 * sq
        fmag = st * xi.square().sum(1).sqrt()
        cap = mu * fn
        slip = fmag > cap
        diss = (fn - fel) * vn * dt + torch.where(slip, cap * (fmag - cap) / st, torch.zeros_like(cap))
        xi = xi * torch.where(slip, cap / torch.clamp(fmag, min=1e-300), torch.ones_like(cap))[:, None]
        f = -fn[:, None] * nrm - st[:, None] * xi
        return f, xi, diss, 0.4 * fel * delta

    def evaluate(self):
        """Forces and torques at the present state; commits histories and breaks."""
        if self.pi is None or self.evals % 20 == 0:
            self.candidates()
        n, x, v, w, r = self.n, self.x, self.v, self.w, self.r
        F = torch.zeros((n, 2), dtype=torch.float64, device=_DEV)
        T = torch.zeros(n, dtype=torch.float64, device=_DEV)
        loss = torch.zeros(n, dtype=torch.float64, device=_DEV)
        self.hertz = torch.zeros(n, dtype=torch.float64, device=_DEV)
        self.bond_el = torch.zeros(n, dtype=torch.float64, device=_DEV)
        perp = lambda a: torch.stack((-a[:, 1], a[:, 0]), 1)  # noqa: E731
        exclude = None
        if self.nb:
            i, j = self.bi, self.bj
            cur = x[j] - x[i]
            u = cur - self.bref
            d = cur.square().sum(1).sqrt()
            ext = (2.0 * (self.bref * u).sum(1) + u.square().sum(1)) / (d + self.bl0)
            g = torch.zeros((n, 4), dtype=torch.float64, device=_DEV)
            m = (u[:, :, None] * self.bref[:, None, :]).reshape(-1, 4)
            g.index_add_(0, i, m).index_add_(0, j, m)
            g = g.reshape(-1, 2, 2) @ self.pinv
            gt = g.transpose(1, 2)
            e = 0.5 * (g + gt + gt @ g)
            s = ((e[:, 0, 0] - e[:, 1, 1]) ** 2 + 4.0 * e[:, 0, 1] ** 2).sqrt()
            fails = (ext / self.bl0 > self.et * self.bf) | (0.5 * (s[i] + s[j]) > self.es * self.bf)
            self.alive = self.alive & ~fails
            a = self.alive & (self.im[i] + self.im[j] > 0)
            i, j, nrm = i[a], j[a], cur[a] / d[a][:, None]
            vrel = v[i] - v[j] + (w[i] * r[i] + w[j] * r[j])[:, None] * perp(nrm)
            vn = (vrel * nrm).sum(1)
            vt = vrel - vn[:, None] * nrm
            dt = self.dt[i]
            us = self.us[a] + vt * dt[:, None]
            us = us - (us * nrm).sum(1)[:, None] * nrm
            self.us[a] = us
            kn, ks, meff = self.kn[a], self.ks[a], 1.0 / (self.im[i] + self.im[j])
            cn, cs = 2.0 * self.zeta[a] * (kn * meff).sqrt(), 2.0 * self.zeta[a] * (ks * meff).sqrt()
            f = (kn * ext[a] - cn * vn)[:, None] * nrm - ks[:, None] * us - cs[:, None] * vt
            cr = nrm[:, 0] * f[:, 1] - nrm[:, 1] * f[:, 0]
            F.index_add_(0, i, f).index_add_(0, j, -f)
            T.index_add_(0, i, r[i] * cr).index_add_(0, j, r[j] * cr)
            loss.index_add_(0, i, (cn * vn**2 + cs * vt.square().sum(1)) * dt)
            self.bond_el.index_add_(0, i, 0.5 * kn * ext[a] ** 2 + 0.5 * ks * us.square().sum(1))
            exclude = (self.bi * n + self.bj)[self.alive]
        i, j = self.pi, self.pj
        d = x[j] - x[i]
        dist = d.square().sum(1).sqrt()
        act = (r[i] + r[j] - dist > 0) & (self.im[i] + self.im[j] > 0)
        if exclude is not None:
            act &= ~torch.isin(i * n + j, exclude)
        i, j, d, dist = i[act], j[act], d[act], dist[act]
        keys = i * n + j
        xi = torch.zeros((len(i), 2), dtype=torch.float64, device=_DEV)
        if len(self.keys) and len(keys):
            at = torch.clamp(torch.searchsorted(self.keys, keys), max=len(self.keys) - 1)
            hit = self.keys[at] == keys
            xi[hit] = self.xi[at[hit]]
        nrm = d / dist[:, None]
        vrel = v[i] - v[j] + (w[i] * r[i] + w[j] * r[j])[:, None] * perp(nrm)
        f, xi, diss, un = self.contact(r[i] + r[j] - dist, nrm, r[i] * r[j] / (r[i] + r[j]),
                                       1.0 / (self.im[i] + self.im[j]), None, vrel, xi, self.e2[i], self.g8[i],
                                       self.damp[i], self.mu[i], self.dt[i])
        self.keys, self.xi = keys, xi
        cr = nrm[:, 0] * f[:, 1] - nrm[:, 1] * f[:, 0]
        F.index_add_(0, i, f).index_add_(0, j, -f)
        T.index_add_(0, i, r[i] * cr).index_add_(0, j, r[j] * cr)
        loss.index_add_(0, i, diss)
        self.hertz.index_add_(0, i, un)
        free = self.im > 0
        for k, (nx, ny) in enumerate(((1.0, 0.0), (-1.0, 0.0), (0.0, 1.0), (0.0, -1.0))):
            gap = x[:, 0] if k == 0 else self.box[:, 0] - x[:, 0] if k == 1 else x[:, 1] if k == 2 else self.box[:, 1] - x[:, 1]
            on = torch.nonzero((r - gap > 0) & ((self.walls >> k) & 1 > 0) & free).flatten()
            new = torch.zeros_like(self.wall_xi[k])
            if len(on):
                nw = torch.tensor([[nx, ny]], dtype=torch.float64, device=_DEV).expand(len(on), 2)
                vc = v[on] - (w[on] * r[on])[:, None] * perp(nw)
                # the wall's side of the contact law: its normal points into the wall
                f, xw, diss, un = self.contact((r - gap)[on], -nw, r[on], 1.0 / self.im[on], None, vc,
                                               self.wall_xi[k, on], self.e2[on], self.g8[on], self.damp[on],
                                               self.muw[on], self.dt[on])
                F.index_add_(0, on, f)
                T.index_add_(0, on, -r[on] * (nx * f[:, 1] - ny * f[:, 0]))
                loss.index_add_(0, on, diss)
                self.hertz.index_add_(0, on, un)
                new[on] = xw
            self.wall_xi[k] = new
        if self.has_ind:
            cen = self.icen + (self.evals * self.dt)[:, None] * self.ivel
            d = x - cen
            dist = d.square().sum(1).sqrt()
            on = torch.nonzero((self.irad > 0) & (self.irad + r - dist > 0) & free).flatten()
            if len(on):
                nw = d[on] / dist[on][:, None]
                delta = (self.irad + r - dist)[on]
                sn = self.e2[on] * (self.irad[on] * r[on] / (self.irad[on] + r[on]) * delta).sqrt()
                fel = (2.0 / 3.0) * sn * delta
                va = -((v[on] - self.ivel[on]) * nw).sum(1)
                fn = torch.clamp(fel + self.damp[on] * (sn / self.im[on]).sqrt() * va, min=0.0)
                F.index_add_(0, on, fn[:, None] * nw)
                loss.index_add_(0, on, (fn - fel) * va * self.dt[on])
                self.hertz.index_add_(0, on, 0.4 * fel * delta)
        F = F + self.m[:, None] * self.g
        self.dissipated += self.sums(loss)
        self.evals += 1
        self.F, self.T = F, T

    def advance(self, steps):
        self.evaluate()
        h = 0.5 * self.dt
        for _ in range(steps):
            self.v = self.v + (h * self.im)[:, None] * self.F
            self.w = self.w + h * self.ii * self.T
            self.x = self.x + self.dt[:, None] * self.v
            self.evaluate()
            self.v = self.v + (h * self.im)[:, None] * self.F
            self.w = self.w + h * self.ii * self.T

    def state(self):
        return dict(pos=self.x, vel=self.v, omega=self.w, force=self.F, torque=self.T)


def _exact_ice2d(case, seed):
    """The reference-mode step, every pair at once: central bonds, penalty contacts, tool, drag, semi-implicit Euler."""
    cfg = DEMConfig(nx=case["nx"], ny=case["ny"], breaking_strain=0.01, shear_breaking_strain=0.02)
    n, dt = cfg.nx * cfg.ny, cfg.recommended_dt
    f8 = dict(dtype=torch.float64, device=_DEV)
    col = torch.arange(cfg.nx, **f8).repeat(cfg.ny)
    row = torch.arange(cfg.ny, **f8).repeat_interleave(cfg.nx)
    x = torch.stack((col - (cfg.nx - 1) / 2, row), 1) * (2 * cfg.radius)
    fixed = (col == 0) | (col == cfg.nx - 1)
    v = _ice2d_velocities(case, seed, n)
    v[fixed] = 0.0
    x0 = x.clone()
    i, j = torch.triu_indices(n, n, offset=1, device=_DEV)
    rest = (x[j] - x[i]).square().sum(1).sqrt()
    bonded = rest <= 2 * cfg.radius * math.sqrt(2) * (1 + 1e-10)
    bi, bj = i[bonded], j[bonded]
    ref = x[bj] - x[bi]
    zeros = lambda *s: torch.zeros(s, **f8)  # noqa: E731
    outer = (ref[:, :, None] * ref[:, None, :]).reshape(-1, 4)
    cov = zeros(n, 4).index_add_(0, bi, outer).index_add_(0, bj, outer)
    pinv = _pinv2(cov)
    alive = bonded.clone()
    mode = torch.zeros(len(i), dtype=torch.uint8, device=_DEV)
    when = torch.full((len(i),), -1.0, **f8)
    top = (cfg.ny - 1) * 2 * cfg.radius + cfg.radius
    tool0 = torch.tensor([0.0, top + cfg.tool_radius + cfg.tool_gap], **f8)
    tool_v = torch.tensor([0.0, -cfg.tool_speed], **f8)
    time = 0.0

    def forces():
        nonlocal alive
        d = x[j] - x[i]
        dist = d.square().sum(1).sqrt()
        nrm = d / dist[:, None]
        ext = dist - rest
        m = ((x[bj] - x[bi])[:, :, None] * ref[:, None, :]).reshape(-1, 4)
        g = zeros(n, 4).index_add_(0, bi, m).index_add_(0, bj, m).reshape(-1, 2, 2) @ pinv
        e = 0.5 * (g.transpose(1, 2) @ g - torch.eye(2, **f8))
        s = ((e[:, 0, 0] - e[:, 1, 1]) ** 2 + 4.0 * e[:, 0, 1] ** 2).sqrt()
        tens = ext / rest > cfg.breaking_strain
        shr = torch.zeros_like(tens)
        shr[bonded] = 0.5 * (s[bi] + s[bj]) > cfg.shear_breaking_strain
        new = alive & (tens | shr)
        mode[new] = (tens[new].to(torch.uint8) + 2 * shr[new].to(torch.uint8))
        when[new] = time
        alive = alive & ~new
        ov = torch.clamp(2 * cfg.radius - dist, min=0.0)
        vn = ((v[j] - v[i]) * nrm).sum(1)
        rep = torch.clamp(cfg.contact_stiffness * ov - cfg.contact_damping * vn, min=0.0)
        rep = torch.where((ov > 0) & ~alive, rep, torch.zeros_like(rep))
        f = torch.where(alive, cfg.bond_stiffness * ext, -rep)[:, None] * nrm
        F = zeros(n, 2).index_add_(0, i, f).index_add_(0, j, -f) - cfg.drag * v
        d = x - (tool0 + time * tool_v)
        dist = d.square().sum(1).sqrt()
        nrm = d / dist[:, None]
        ov = torch.clamp(cfg.radius + cfg.tool_radius - dist, min=0.0)
        mag = torch.clamp(cfg.contact_stiffness * ov - cfg.contact_damping * ((v - tool_v) * nrm).sum(1), min=0.0)
        ft = torch.where(ov > 0, mag, torch.zeros_like(mag))[:, None] * nrm
        return F + ft, -ft.sum(0)

    for _ in range(case["steps"]):
        F, _r = forces()
        v = v + dt * F / cfg.mass
        v[fixed] = 0.0
        x = x + dt * v
        x[fixed] = x0[fixed]
        time += dt
    F, reaction = forces()
    return dict(positions=x, velocities=v, force=F, reaction=reaction, alive=alive, failure_mode=mode,
                failure_time=when)


def _exact_ice3d(case, seed):
    """The first steps of an intact 3-D specimen that the indenter has not reached: bonds, drag, Euler."""
    cfg = _ice3d_config(case)
    f8 = dict(dtype=torch.float64, device=_DEV)
    probe = IceDEM3D(cfg)  # the lattice, its bonds and the time step: inputs of the pass
    x, fixed, dt = probe.initial_positions.clone(), probe.fixed, probe.dt
    x0 = x.clone()
    v = _ice3d_velocities(seed, probe)
    i, j = probe.pairs[probe.bonded].T
    rest = (x[j] - x[i]).square().sum(1).sqrt()
    for _ in range(case["steps"]):
        d = x[j] - x[i]
        dist = d.square().sum(1).sqrt()
        if bool((dist / rest - 1.0 > cfg.breaking_strain).any()):
            return None
        f = (cfg.bond_stiffness * (dist - rest) / dist)[:, None] * d
        F = torch.zeros((len(x), 3), **f8).index_add_(0, i, f).index_add_(0, j, -f) - cfg.drag * v
        v = v + dt * F / cfg.mass
        v[fixed] = 0.0
        x = x + dt * v
        x[fixed] = x0[fixed]
    return dict(positions=x, velocities=v, alive=None, failure_mode=None, reaction=None)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("gas", "bed", "sheet"):
        if case["nx"] * case["ny"] * case["steps"] > 6e8:
            return None
        d = _Discs([_hm_case(case, seed)])
        d.advance(case["steps"])
        return d.state()
    if kind == "batch":
        insts = _batch_instances(case, seed)
        d = _Discs([(replace(i.config, precision=case["precision"]), i.state, i.bonds, i.strength) for i in insts])
        d.advance(case["steps"])
        s = d.state()
        out = {k: None for k in _LEDGER}
        free = d.im > 0
        inertia = torch.where(free, 1.0 / d.ii, torch.zeros_like(d.ii))
        out["kinetic"] = d.sums(0.5 * d.m * d.v.square().sum(1) + 0.5 * inertia * d.w**2)
        out["potential"] = d.sums(-d.m * (d.x * d.g).sum(1))
        out["hertz"], out["bond_elastic"] = d.sums(d.hertz), d.sums(d.bond_el)
        out["dissipated"] = d.dissipated
        out = {k: None if u is None else u.cpu().numpy() for k, u in out.items()}
        for at in (0, -1):
            a, b = int(d.first[:-1][at]), int(d.first[1:][at])
            out.update({f"{k}_{at}": u[a:b].cpu().numpy() for k, u in s.items()})
        return out
    return _exact_ice2d(case, seed) if kind == "ice2d" else _exact_ice3d(case, seed)
