"""The work a user of this framework has it do, as timed cases.

Every case goes through the public Python API (`CryoSPH`): a tank or a dam
break is loaded, stepped, and its state read back -- as a simulation loop that
writes a frame every few steps does.  Sizes come from this repository's
benchmark and tests (the closed LN2 cylinder, the SPHERIC dam break, the LH2
sphere, the tank ensemble, the boil-off window of the adjoint) and from odd
lattice spacings between and beyond them.

A case is a dict of plain values; `prepare` loads the solver from it and a
seed, `run` makes one pass, `work` counts what the pass cannot do without and
`exact` restates the dam-break cases in 64 bits.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "microgravity-cryogenic-multi-phase-sph-solver_b200"))
import CryoSPH as cs  # noqa: E402


# --------------------------------------------------------------------- cases
def listed():
    return [
        # a controller's loop on a small tank: per pass one frame input, one
        # step, the blocking diagnostics and eight pressure sensors; latency
        # and launches count, nothing else
        dict(name="control loop 27k", kind="loop", dx=0.05, arith="exact"),
        # the smallest tank run in earnest, the constructor's defaults (vented,
        # Lee phase change, CSF, heat), a frame every 20 steps
        dict(name="vented box 4k", kind="tank", shape="box", size=0.04, aspect=1.0, dx=0.004, fill=0.5,
             fluid="nitrogen", closed=False, heater=0.0, arith="exact", steps=20),
        # the reference's headline tank: closed LN2 cylinder at 4 mm with a heater
        dict(name="heated cylinder 26k", kind="tank", shape="cylinder", size=0.05, aspect=2.4, dx=0.004, fill=0.5,
             fluid="nitrogen", closed=True, heater=20.0, arith="exact", steps=20),
        # the same tank refined, in the fast arithmetic, particles followed by id
        dict(name="cylinder 91k fast", kind="tank", shape="cylinder", size=0.05, aspect=2.4, dx=0.00247, fill=0.6,
             fluid="oxygen", closed=True, heater=0.0, arith="fast", steps=20),
        # the benchmark's dam break (203 662 particles), fast and exact
        dict(name="dam break 204k fast", kind="dam", dx=0.02, arith="fast", no_slip=False, sps=False, steps=40),
        dict(name="dam break 204k", kind="dam", dx=0.02, arith="exact", no_slip=False, sps=False, steps=40),
        # a finer dam break with no-slip walls and sub-particle stresses, odd spacing
        dict(name="dam break 503k fast", kind="dam", dx=0.0139, arith="fast", no_slip=True, sps=True, steps=20),
        # the two-phase LH2 sphere: a million particles, fast; four million, exact
        dict(name="sphere 1.06M fast", kind="tank", shape="sphere", size=0.5, aspect=1.0, dx=0.0083, fill=0.5,
             fluid="hydrogen", closed=True, heater=0.0, arith="fast", steps=12),
        dict(name="sphere 4.08M", kind="tank", shape="sphere", size=0.5, aspect=1.0, dx=0.0052, fill=0.5,
             fluid="hydrogen", closed=True, heater=0.0, arith="exact", steps=8),
        # a design study: many small tanks side by side in one ensemble
        dict(name="ensemble of 20", kind="ensemble", tanks=20, smallest=4000, largest=60000, arith="exact", steps=10),
        # forward and backward through a differentiated window of the boil-off tank
        dict(name="adjoint window 41k", kind="adjoint", dx=0.0068, steps=20, every=10),
        # a restart loop: host arrays (NumPy's float64) loaded, a few steps, the state read back
        dict(name="restart 204k", kind="restart", dx=0.02, arith="exact", steps=4),
    ]


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm."""
    def spread(lo, hi):
        return float(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["tank", "tank", "tank", "dam", "dam", "loop", "ensemble", "adjoint", "restart"])
    if kind == "tank":
        shape = rng.choice(["box", "cylinder", "sphere", "capsule"])
        size = spread(0.03, 0.4)
        aspect = 1.0 if shape in ("box", "sphere") else round(rng.uniform(1.0, 2.5), 3)
        cells = spread(14.0, 96.0)  # particles across
        across = size if shape == "box" else 2.0 * size
        return dict(kind="tank", shape=shape, size=size, aspect=aspect, dx=across / cells,
                    fill=round(rng.uniform(0.2, 0.8), 3), fluid=rng.choice(["nitrogen", "oxygen", "methane", "hydrogen"]),
                    closed=rng.random() < 0.7, heater=rng.choice([0.0, 0.0, 20.0]), arith=rng.choice(["exact", "fast"]),
                    steps=rng.choice([10, 15, 20]))
    if kind == "dam":
        no_slip = rng.random() < 0.4
        return dict(kind="dam", dx=spread(0.0135, 0.06), arith=rng.choice(["exact", "fast"]), no_slip=no_slip,
                    sps=no_slip and rng.random() < 0.5, steps=rng.choice([10, 20, 30]))
    if kind == "loop":
        return dict(kind="loop", dx=spread(0.03, 0.08), arith="exact")
    if kind == "ensemble":
        return dict(kind="ensemble", tanks=rng.randint(3, 24), smallest=3000, largest=int(spread(8000, 60000)),
                    arith="exact", steps=rng.choice([5, 10]))
    if kind == "adjoint":
        return dict(kind="adjoint", dx=spread(0.0062, 0.012), steps=rng.choice([8, 14, 20]), every=rng.choice([5, 10]))
    return dict(kind="restart", dx=spread(0.018, 0.06), arith="exact", steps=rng.randint(1, 6))


# -------------------------------------------------------------------- inputs
def _arith(solver, case):
    if case["arith"] == "fast":
        solver.field_arithmetic = cs.FieldArithmetic.Fast
    return solver


def _dam_config(case):
    """SPHERIC Test 2: continuity density, no surface tension, no heat."""
    cfg = cs.SolverConfig()
    cfg.dx = case["dx"]
    cfg.gravity = (0.0, 0.0, -9.81)
    cfg.surface_tension = type(cfg.surface_tension)(0)
    cfg.thermal = False
    cfg.phase_change = False
    cfg.density_mode = type(cfg.density_mode)(1)
    cfg.velocity_scale = (2 * 9.81 * 0.55) ** 0.5
    cfg.artificial_viscosity = 0.02
    cfg.delta_sph = 0.1
    cfg.no_slip = bool(case.get("no_slip", False))
    cfg.sps_turbulence = bool(case.get("sps", False))
    return cfg


def _dam_fluid():
    water = cs.FluidProperties.water()
    water.mu_liquid = 1.0e-3
    return water


@functools.lru_cache(maxsize=4)
def _dam_lattice(dx):
    """The tank with its obstacle, and the water column 1.228 m long and 0.55 m high at the far end."""
    box = (0.161, 0.403, 0.161)
    tank = cs.Difference(cs.Translated(cs.BoxTank(3.22, 1.0, 1.0), (1.61, 0.0, 0.5)),
                         cs.Translated(cs.BoxTank(*box), (0.744 - box[0] / 2, 0.0, box[2] / 2)))
    fill = cs.FillSpec()
    fill.mode = cs.FillMode.Full
    p = cs.tank_particles(tank, _dam_fluid(), dx, fill)
    x = np.asarray(p["position"])
    keep = (p["phase"] == 2) | ((x[:, 0] > 3.22 - 1.228) & (x[:, 2] < 0.55))
    return {k: np.asarray(v)[keep] for k, v in p.items()}


def _dam_particles(dx, seed):
    """The column on a jittered lattice, already moving: a collapsing flow
    (u, w) = s (x - 3.22, -z), s of the seed, walls at rest."""
    rng = np.random.default_rng(seed)
    p = dict(_dam_lattice(dx))
    fluid = p["phase"] != 2
    x = p["position"].astype(np.float64)
    x[fluid] += rng.uniform(-0.05 * dx, 0.05 * dx, size=(int(fluid.sum()), 3))
    s = float(rng.uniform(0.5, 1.5))
    v = np.zeros_like(x)
    v[fluid, 0] = s * (x[fluid, 0] - 3.22)
    v[fluid, 2] = -s * x[fluid, 2]
    p["position"] = x.astype(np.float32)
    p["velocity"] = v.astype(np.float32)
    return p


def _dam_domain(dx):
    pad = 4 * dx
    return (-pad, -0.5 - pad, -pad), (3.22 + pad, 0.5 + pad, 1.0 + pad)


def _load(solver, p, lo, hi):
    solver.set_particles(p["position"], p["mass"], p["density"], p["temperature"], p["phase"], domain_lo=lo,
                         domain_hi=hi, velocity=p["velocity"], normal=p["normal"], flags=p["flags"])


def _dam_solver(case, seed):
    s = _arith(cs.Solver(_dam_config(case), _dam_fluid()), case)
    _load(s, _dam_particles(case["dx"], seed), *_dam_domain(case["dx"]))
    return s


_FLUIDS = {"nitrogen": cs.FluidProperties.liquid_nitrogen, "oxygen": cs.FluidProperties.liquid_oxygen,
           "methane": cs.FluidProperties.liquid_methane, "hydrogen": cs.FluidProperties.liquid_hydrogen}


def _geometry(shape, size, aspect):
    if shape == "box":
        return cs.BoxTank(size, size, size)
    if shape == "sphere":
        return cs.SphereTank(size)
    if shape == "capsule":
        return cs.CapsuleTank(size, size * aspect)
    return cs.CylinderTank(size, size * aspect)


def _fill(case):
    fill = cs.FillSpec()
    fill.fill_fraction = case["fill"]
    return fill


def _tank_solver(case, seed):
    """A two-phase tank at 1e-4 g, a superheated and jittered lattice, under a lateral pulse."""
    fluid = _FLUIDS[case["fluid"]]()
    cfg = cs.SolverConfig()
    cfg.dx = case["dx"]
    cfg.gravity = (0.0, 0.0, -9.81e-4)
    cfg.thermo_mode = cs.TankThermoMode.Closed if case["closed"] else cs.TankThermoMode.Vented
    cfg.heater_power = case["heater"]
    fill = _fill(case)
    fill.T_liquid = fluid.T_sat + 1.0
    s = _arith(cs.Solver(cfg, fluid), case)
    s.build_tank(_geometry(case["shape"], case["size"], case["aspect"]), fill)
    s.jitter_fluid(0.05 * case["dx"], int(seed))
    pulse = 0.1 * float(np.random.default_rng(seed).uniform(0.2, 1.0))
    s.set_maneuver(cs.ManeuverProfile([0.0, 0.01, 0.05, 0.06],
                                      np.array([[0, 0, 0], [pulse, 0, 0], [pulse, 0, 0], [0, 0, 0]], np.float64)))
    return s


def _ensemble_tanks(case):
    """Cylinders and spheres whose particle counts run from the smallest to the largest over their logarithm."""
    tanks = []
    for k in range(case["tanks"]):
        f = k / max(1, case["tanks"] - 1)
        n = case["smallest"] * (case["largest"] / case["smallest"]) ** f
        sphere = k % 2 == 0
        size = 0.03 + 0.27 * ((k * 7) % case["tanks"]) / case["tanks"]
        aspect = 1.0 if sphere else 2.0 + 0.1 * (k % 20)
        vol = 4.0 / 3.0 * math.pi * size ** 3 if sphere else math.pi * aspect * size ** 3
        area = 4.0 * math.pi * size ** 2 if sphere else 2.0 * math.pi * size * size * (aspect + 1.0)
        lo, hi = 1e-5, 1.0
        for _ in range(60):  # interior lattice and three wall layers make up n
            dx = math.sqrt(lo * hi)
            lo, hi = (dx, hi) if vol / dx ** 3 + 3.0 * area / dx ** 2 > n else (lo, dx)
        tanks.append(dict(shape="sphere" if sphere else "cylinder", size=size, aspect=aspect, dx=math.sqrt(lo * hi),
                          fill=0.2 + 0.6 * ((k * 3) % 11) / 11.0, fluid=["nitrogen", "oxygen", "methane"][k % 3],
                          closed=True, heater=0.0, arith=case["arith"]))
    return tanks


def _boiloff_solver(case, seed):
    """The differentiated workload: closed LN2 cylinder, 2 K superheat, 20 W
    heater, a fixed step and a pinned sound speed, no splits or merges."""
    fluid = cs.FluidProperties.liquid_nitrogen()
    cfg = cs.SolverConfig()
    cfg.dx = case["dx"]
    cfg.gravity = (0.0, 0.0, -9.81e-4)
    cfg.thermo_mode = cs.TankThermoMode.Closed
    cfg.heater_power = 20.0
    cfg.lee_evaporation = 5.0
    cfg.lee_condensation = 5.0
    cfg.fixed_dt = 1e-3
    cfg.sound_speed = 0.5
    cfg.split_ratio = 1e3
    cfg.merge_ratio = 0.0
    s = cs.Solver(cfg, fluid)
    fill = cs.FillSpec()
    fill.fill_fraction = 0.5
    fill.T_liquid = fluid.T_sat + 2.0
    s.build_tank(cs.CylinderTank(0.1, 0.25), fill)
    s.jitter_fluid(0.02 * case["dx"], int(seed))
    return s


_SENSORS = np.array([(0.744, y, z) for y in (-0.05, 0.05) for z in (0.021, 0.101)]
                    + [(x, 0.0, 0.1) for x in (2.2, 2.5, 2.8, 3.1)], np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dam":
        return dict(case=case, solver=_dam_solver(case, seed))
    if kind == "loop":
        return dict(case=case, solver=_dam_solver(case, seed), acc=float(np.random.default_rng(seed).uniform(0.1, 1.0)))
    if kind == "tank":
        return dict(case=case, solver=_tank_solver(case, seed))
    if kind == "ensemble":
        e = cs.Ensemble()
        members = [_tank_solver(t, seed + 1000 * k) for k, t in enumerate(_ensemble_tanks(case))]
        for m in members:
            e.add(m)
        return dict(case=case, ensemble=e, members=members)
    if kind == "adjoint":
        seeds = np.random.default_rng(seed).uniform(0.5, 1.5, 7)
        seeds[6] *= 1e-4  # Pa against N s
        return dict(case=case, solver=_boiloff_solver(case, seed), weights=[float(w) for w in seeds])
    # restart: the arrays in host memory are the input, the solver is kept
    p = _dam_particles(case["dx"], seed)
    p = {k: v.astype(np.float64) if v.dtype == np.float32 else v for k, v in p.items()}
    return dict(case=case, solver=_arith(cs.Solver(_dam_config(case), _dam_fluid()), case), particles=p,
                domain=_dam_domain(case["dx"]))


# --------------------------------------------------------------------- a pass
def _by_id(p, *fields):
    """The state as tensors with one row per particle id (the solver keeps its arrays in cell order)."""
    rows = int(p["id"].max()) + 1
    ids = torch.from_numpy(p["id"].view(np.int32)).cuda().long()
    out = {}
    for f in fields:
        a = torch.from_numpy(p[f]).cuda()
        t = torch.zeros((rows, *a.shape[1:]), dtype=a.dtype, device=a.device)
        t[ids] = a
        out[f] = t
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        state["ensemble"].run_steps(case["steps"])
        ps = [m.particles() for m in state["members"]]
        return {f: np.concatenate([p[f] for p in ps]) for f in ("position", "velocity", "temperature", "mass")}
    s = state["solver"]
    if kind == "loop":
        s.set_frame_motion(acceleration=(state["acc"], 0.0, 0.0))
        s.step()
        d = s.diagnostics()
        return {"pressure": s.probe_pressure(_SENSORS), "mass": d.mass_liquid, "kinetic_energy": d.kinetic_energy,
                "com": np.array(d.liquid_com), "momentum": np.array(d.liquid_momentum),
                "force": np.array(d.slosh_force, np.float32), "moment": np.array(d.slosh_moment, np.float32)}
    if kind == "adjoint":
        objectives = s.adjoint_forward(case["steps"], case["every"])
        return {"objectives": objectives, **s.adjoint_backward(state["weights"])}
    if kind == "restart":
        _load(s, state["particles"], *state["domain"])
    s.run_steps(case["steps"])
    p = s.particles()
    if kind in ("dam", "restart"):  # particles followed by id
        return _by_id(p, "position", "velocity", "density")
    if case["arith"] == "fast":
        return _by_id(p, "position", "velocity", "temperature", "mass")
    return {f: p[f] for f in ("position", "velocity", "density", "temperature", "mass", "phase", "id")}


# ----------------------------------------------------------------------- work
@functools.lru_cache(maxsize=64)
def _tank_counts(shape, size, aspect, dx, fill, fluid):
    f = cs.FillSpec()
    f.fill_fraction = fill
    phase = cs.tank_particles(_geometry(shape, size, aspect), _FLUIDS[fluid](), dx, f)["phase"]
    return int((phase != 2).sum()), int((phase == 2).sum())


def _counts(case):
    kind = case["kind"]
    if kind == "tank":
        return [_tank_counts(case["shape"], case["size"], case["aspect"], case["dx"], case["fill"], case["fluid"])]
    if kind == "ensemble":
        return [_tank_counts(t["shape"], t["size"], t["aspect"], t["dx"], t["fill"], t["fluid"])
                for t in _ensemble_tanks(case)]
    if kind == "adjoint":
        return [_tank_counts("cylinder", 0.1, 2.5, case["dx"], 0.5, "nitrogen")]
    phase = _dam_lattice(case["dx"])["phase"]
    return [(int((phase != 2).sum()), int((phase == 2).sum()))]


def work(case):
    """A step reads and writes each particle's state once (84 bytes; a wall's
    36) and evaluates each pair of a fluid particle's 73 neighbours (the
    support sphere of 2.6 spacings) at about 60 operations, twice that with
    surface tension, heat and phase change; the state goes to the host once."""
    nf, nw = (sum(c[k] for c in _counts(case)) for k in (0, 1))
    two_phase = case["kind"] in ("tank", "ensemble", "adjoint")
    steps = case.get("steps", 1) * (3 if case["kind"] == "adjoint" else 1)  # forward, recomputation, reverse
    out = 0 if case["kind"] in ("loop", "adjoint") else 58 * (nf + nw)
    load = 58 * (nf + nw) if case["kind"] == "restart" else 0
    return {"bytes": steps * (168 * nf + 72 * nw) + out + load, "flops": steps * nf * 73 * (120 if two_phase else 60)}


# -------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """The dam-break passes (free-slip, no sub-particle stresses) in 64 bits,
    rows by particle id.  The two-phase tanks have none: their passes carry
    on/off decisions (interface normals, Lee caps, rebalance) that a 64-bit run
    takes otherwise within a few steps."""
    if case["kind"] not in ("dam", "restart") or case.get("no_slip"):
        return None
    x, v, rho = _dam64(case, seed, case["steps"])
    return {"position": x, "velocity": v, "density": rho}


def _pairs(x, i_sel, j_sel, support, cell):
    """(i, j) of every i in i_sel and j in j_sel closer than `support`, i == j included."""
    lo = x.min(0).values - cell
    c = ((x - lo) / cell).floor().long()
    dims = (c.max(0).values + 2).tolist()
    key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
    kj, order = key[j_sel].sort()
    sj = j_sel[order]
    count = torch.zeros(dims[0] * dims[1] * dims[2] + 1, dtype=torch.long, device=x.device)
    count.index_add_(0, kj + 1, torch.ones_like(kj))
    begin = count.cumsum(0)
    found_i, found_j = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            k0 = key[i_sel] + (dz * dims[1] + dy) * dims[0]
            s, e = begin[k0 - 1], begin[k0 + 2]
            n = e - s
            ii = torch.repeat_interleave(i_sel, n)
            first = torch.repeat_interleave(s - (n.cumsum(0) - n), n)
            jj = sj[first + torch.arange(ii.numel(), device=x.device)]
            near = (x[ii] - x[jj]).square().sum(1) < support * support
            found_i.append(ii[near])
            found_j.append(jj[near])
    return torch.cat(found_i), torch.cat(found_j)


def _dam64(case, seed, steps):
    f8 = dict(dtype=torch.float64, device="cuda")
    f32 = np.float32
    p = _dam_particles(case["dx"], seed)
    x = torch.from_numpy(p["position"]).cuda().double()
    v = torch.from_numpy(p["velocity"]).cuda().double()
    rho = torch.from_numpy(np.asarray(p["density"], f32)).cuda().double()
    wall = torch.from_numpy(p["phase"] == 2).cuda()
    fl, wl = (~wall).nonzero()[:, 0], wall.nonzero()[:, 0]
    n = x.shape[0]
    dx = float(f32(case["dx"]))
    h = float(f32(1.3)) * dx
    support, norm = 2.0 * h, 21.0 / (16.0 * math.pi * h ** 3)
    rho0, mu = float(f32(998.2)), float(f32(1.0e-3))
    c0 = 10.0 * float(f32((2 * 9.81 * 0.55) ** 0.5))
    B = rho0 * c0 * c0 / 7.0
    g = torch.tensor([0.0, 0.0, -float(f32(9.81))], **f8)
    av, delta = float(f32(0.02)), float(f32(0.1))

    def W(r):
        q = r / h
        t = (1.0 - 0.5 * q).clamp(min=0.0)
        return norm * t ** 4 * (2.0 * q + 1.0)

    k = torch.arange(-3, 4, **f8)
    vol0 = 1.0 / W(dx * torch.stack(torch.meshgrid(k, k, k, indexing="ij")).square().sum(0).sqrt()).sum()

    def add(i, val):
        out = torch.zeros((n, *val.shape[1:]), **f8)
        return out.index_add_(0, i, val)

    def rates(x, v, rho, m, dt):
        """Accelerations and density rates of the fluid; the maxima of the next step size."""
        press = B * ((rho / rho0) ** 7 - 1.0)
        i, j = _pairs(x, wl, fl, support, support)  # walls: Shepard pressure with the hydrostatic term
        r = (x[i] - x[j])
        w = W(r.square().sum(1).sqrt())
        sw = add(i, w)
        pw = add(i, press[j] * w + (r @ g) * rho[j] * w) / sw.clamp(min=1e-300)
        press = torch.where(wall, torch.where(sw > 0, pw, torch.zeros_like(pw)), press)
        i, j = _pairs(x, fl, torch.arange(n, device=x.device), support, support)
        apart = i != j
        i, j = i[apart], j[apart]
        rij = x[i] - x[j]
        r2 = rij.square().sum(1)
        r = r2.sqrt()
        t = 1.0 - 0.5 * r / h
        gw = rij * (-5.0 * norm / (h * h) * t ** 3)[:, None]  # dW/dr / r
        rmin = torch.full((n,), support, **f8).scatter_reduce(0, i, r, "amin")
        a = torch.zeros_like(x) + g
        drho = torch.zeros(n, **f8)
        Vi = m / rho
        w_ = wall[j]
        # walls
        ii, jj, rw, gww = i[w_], j[w_], r[w_], gw[w_]
        force = add(ii, -gww * ((Vi[ii] ** 2 + vol0 ** 2) * 0.5 * (press[ii] + press[jj]))[:, None])
        guard = 0.6 * dx
        nn = rij[w_] / rw[:, None]
        qg = (1.0 - rw / guard).clamp(min=0.0)
        push = 4.0 * c0 * c0 * qg * qg / guard
        if dt > 0:
            vn = (v[ii] * nn).sum(1)
            push = push - torch.where((qg > 0) & (vn < 0), qg * vn / dt, torch.zeros_like(vn))
        a += add(ii, nn * push[:, None])
        div = add(ii, vol0 * (v[ii] * gww).sum(1))
        # fluid
        f_ = ~w_
        ii, jj, rij, r2, r, gw = i[f_], j[f_], rij[f_], r2[f_], r[f_], gw[f_]
        vs = Vi[ii] ** 2 + Vi[jj] ** 2
        force += add(ii, -gw * (vs * (rho[jj] * press[ii] + rho[ii] * press[jj]) / (rho[ii] + rho[jj]))[:, None])
        vij = v[ii] - v[jj]
        force += add(ii, vij * (vs * mu * (gw * rij).sum(1) / r2)[:, None])
        vr = (vij * rij).sum(1)
        mu_ij = h * vr.clamp(max=0.0) / (r2 + 0.01 * h * h)
        a += add(ii, -gw * (m[jj] * -av * c0 * mu_ij / (0.5 * (rho[ii] + rho[jj])))[:, None])
        div += add(ii, Vi[jj] * (vij * gw).sum(1))
        diff = add(ii, -Vi[jj] * 2.0 * (rho[jj] - rho[ii]) * (rij * gw).sum(1) / (r2 + 0.01 * h * h))
        a += force / m[:, None]
        drho = rho * div + delta * h * c0 * diff
        a[wl] = 0.0
        drho[wl] = 0.0
        vmax = v[fl].norm(dim=1).max().item()
        amax = a[fl].norm(dim=1).max().item()
        ratio = (0.5 * dx / rmin[fl].clamp(min=0.05 * dx)).max().item()
        return a, drho, max(1.0, ratio), vmax, amax

    i, j = _pairs(x, fl, torch.arange(n, device=x.device), support, support)
    sigma = add(i, W((x[i] - x[j]).norm(dim=1)))
    m = torch.where(wall, torch.ones_like(rho), rho / sigma.clamp(min=1e-300))
    a, drho, ratio, vmax, amax = rates(x, v, rho, m, 0.0)
    for _ in range(steps):
        dt = 0.25 * h / ((c0 + vmax) * ratio)
        dt = min(dt, 0.125 * h * h / (mu / rho0))
        if amax > 0:
            dt = min(dt, 0.25 * math.sqrt(h / amax))
        dt = max(1e-9, min(dt, 1e-2))
        v = v + 0.5 * dt * a
        x = x + dt * v
        rho = rho + dt * drho
        a, drho, ratio, vmax, amax = rates(x, v, rho, m, dt)
        v = v + 0.5 * dt * a
    # a wall's density is the Shepard mean of the fluid it sees
    i, j = _pairs(x, wl, fl, support, support)
    w = W((x[i] - x[j]).norm(dim=1))
    sw, srho = add(i, w), add(i, w * rho[j])
    rho = torch.where(wall, torch.where(sw > 0, srho / sw.clamp(min=1e-300), torch.full_like(rho, rho0)), rho)
    return x, v, rho
