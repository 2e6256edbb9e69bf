"""Routes of the neighbour passes that only some tanks take: particles the
passes leave out, overflowing lists in the one-thread build, the shapes an
ensemble chooses.  Every comparison is bit for bit."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import CryoSPH as cs
import cryo_cabi as cabi
from test_pass_shapes_gpu import OTHER_ROUTE, big_tank

pytestmark = pytest.mark.gpu

DX = 0.004
STATE = ("x", "v", "rho", "T", "m", "p", "a", "sigma", "nrm", "alpha", "kappa", "fw", "mw", "id", "phase", "flags")


def same(a, b):
    for f in a:
        assert np.array_equal(np.asarray(a[f]).view(np.uint8), np.asarray(b[f]).view(np.uint8)), f


def box(cells, vapour=True):
    fluid = cs.FluidProperties.liquid_nitrogen()
    geometry = cs.BoxTank(cells * DX, cells * DX, cells * DX)
    fill = cs.FillSpec()
    fill.fill_fraction, fill.include_vapor, fill.T_liquid, fill.heater_zmax = 0.5, vapour, fluid.T_sat + 2.0, 0.01
    p = cs.tank_particles(geometry, fluid, DX, fill)
    p["position"] = p["position"] + np.random.default_rng(3).uniform(-4e-4, 4e-4, p["position"].shape).astype(np.float32)
    return p, cs.tank_domain(geometry, DX, 3)


def context(p, domain, arithmetic=0, lists=1, fluid=cabi.FLUID_LN2, **kw):
    g = cabi.Context(cabi.py_config(dx=DX, gravity=(0.05, 0, -0.01), thermo_mode=1, **kw), cabi.py_fluid(fluid))
    g.set_neighbor_mode(lists)
    g.set_field_arithmetic(arithmetic)
    g.set_particles({"x": p["position"], "m": p["mass"], "rho": p["density"], "T": p["temperature"],
                     "phase": p["phase"], "nrm": p["normal"], "flags": p["flags"]}, *domain)
    return g


# 20: lanes in every pass; 54: 157 464 fluid particles, a thread per particle in every pass
@pytest.mark.parametrize("cells", [20, 54])
@pytest.mark.parametrize("kw", [dict(), dict(particle_shifting=1), dict(heater_power=20.0, wetting_model=2),
                                dict(particle_shifting=1, split_ratio=1.02, merge_ratio=0.9)])
def test_particles_left_out_change_nothing(cuda_device, cells, kw):
    """Without lists no pass leaves a particle out; with them the interface
    pass skips the bulk and the phase-change pass the cells no source marked."""
    p, domain = box(cells)
    out = []
    for lists in (1, 0):
        g = context(p, domain, lists=lists, **kw)
        g.step(4)
        out.append({f: g.field(f) for f in STATE})
        out[-1]["evaporated"] = np.array([g.diagnostics().as_dict()[k] for k in ("mass_liquid", "mass_vapor")])
    same(*out)


@pytest.mark.parametrize("n", [70_001, 130_003])
@pytest.mark.parametrize("vapour", [False, True])
def test_overflowing_lists_of_the_one_thread_build(cuda_device, n, vapour):
    """A clump of over 128 neighbours among more particles than share lanes in the build."""
    lo, hi = (0.0, 0.0, 0.0), (0.4, 0.3, 0.2)
    rng = np.random.default_rng(n)
    x = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    x[:700] = rng.uniform((0.1, 0.1, 0.1), (0.112, 0.112, 0.112), (700, 3)).astype(np.float32)
    phase = np.zeros(n, np.uint8)
    phase[::7] = 2
    if vapour:
        phase[1:350:3] = 1
    out = []
    for lists in (1, 0):
        g = cabi.Context(cabi.py_config(dx=0.004, gravity=(0, 0, -1.0), velocity_scale=1.0, thermo_mode=1,
                                        fixed_dt=1e-6, phase_change=int(vapour), surface_tension=int(vapour),
                                        split_ratio=1e3),
                         cabi.py_fluid(cabi.FLUID_H2O))
        g.set_neighbor_mode(lists)
        g.set_particles({"x": x, "m": np.full(n, 1e-3, np.float32), "rho": np.full(n, 1000, np.float32),
                         "T": np.full(n, 374, np.float32), "phase": phase}, lo, hi)
        g.step(2)
        if lists:
            counts = g.neighbor_lists()[0]
            assert len(counts) > 60_000 and counts.max() > 128 and (counts <= 128).any()
        out.append({f: g.field(f) for f in STATE})
    same(*out)


def shapes_of(run):
    """Names of the kernels launched by run().  A capture can miss the first
    kernels after it opens, hence several."""
    torch.zeros(1, device="cuda")
    names = set()
    for _ in range(4):
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            run()
            torch.cuda.synchronize()
        names |= {e.key for e in prof.key_averages()}
    if not any("k_forces_t" in k for k in names):
        pytest.skip("the profiler records no kernels here")
    return names


def test_an_ensemble_changes_the_shapes_and_no_bit(cuda_device):
    """A shifted two-phase tank, alone with lanes in every pass and beside a
    tank that fills the chip with a thread per particle."""
    def make():
        cfg = cs.SolverConfig()
        cfg.dx, cfg.particle_shifting, cfg.thermo_mode = DX, True, cs.TankThermoMode.Closed
        fluid = cs.FluidProperties.liquid_nitrogen()
        fill = cs.FillSpec()
        fill.fill_fraction, fill.T_liquid = 0.5, fluid.T_sat + 3.0
        s = cs.Solver(cfg, fluid)
        s.build_tank(cs.BoxTank(0.06, 0.06, 0.06), fill)
        s.jitter_fluid(0.0003, 5)
        return s

    water, p, (lo, hi) = big_tank()
    cfg = cs.SolverConfig()
    cfg.dx = DX
    filler = cs.Solver(cfg, water)
    filler.set_particles(p["position"], p["mass"], p["density"], p["temperature"], p["phase"], domain_lo=lo,
                         domain_hi=hi, normal=p["normal"], flags=p["flags"])
    crowd, alone, beside = cs.Ensemble(0), make(), make()
    crowd.add(filler)
    crowd.add(beside)
    alone.run_steps(6)
    crowd.run_steps(6)
    a, b = alone.particles(), beside.particles()
    same(a, b)
    assert alone.diagnostics().as_dict() == beside.diagnostics().as_dict()
    with_lanes = shapes_of(lambda: (alone.run_steps(2), alone.diagnostics()))
    with_threads = shapes_of(lambda: (crowd.run_steps(2), crowd.diagnostics()))
    for name, lanes, threads in (("k_density", "lanes::", "exact::"), ("k_wall", "lanes::", "exact::"),
                                 ("k_interface", "lanes::", "exact::"), ("k_forces_t", "lanes::", "exact::"),
                                 ("k_build_lists", "<4>", "<1>"), ("k_pc_normalize", "<8>", "<1>"),
                                 ("k_pc_apply", "<8>", "<1>"), ("k_rebalance1", "<8>", "<1>")):
        a = [k for k in with_lanes if name in k]
        b = [k for k in with_threads if name in k]
        assert a and all(lanes in k and threads not in k for k in a), (name, a)
        assert b and all(threads in k and lanes not in k for k in b), (name, b)


@pytest.mark.parametrize("base,other", [(b, o) for b, o, arithmetics in OTHER_ROUTE if 1 in arithmetics])
@pytest.mark.parametrize("clump", [0, 700])
def test_fast_force_pass_without_the_rarer_options(cuda_device, base, other, clump):
    """The fast instances also agree where a particle searches the cells:
    without lists, and with more neighbours than a list holds."""
    base = dict(base)
    p, domain = box(24, vapour=base["surface_tension"] == 1)
    x, T = p["position"].copy(), np.full(len(p["mass"]), base.pop("T", 300.0), np.float32)
    fluid = np.flatnonzero(p["phase"] != 2)[:clump]
    x[fluid] = np.random.default_rng(2).uniform(-0.005, 0.005, (clump, 3)).astype(np.float32) + x.mean(0)
    out = []
    for extra in ({}, other):
        g = context(dict(p, position=x, temperature=T), domain, 1, int(clump > 0), cabi.FLUID_H2O, phase_change=0,
                    transport_interface_only=0, fixed_dt=1e-6, **base, **extra)
        g.step(2)
        if clump:
            assert g.neighbor_lists()[0].max() > 128
        out.append({f: g.field(f) for f in ("x", "v", "rho", "T", "a", "ab", "drho", "dTdt", "fw", "mw")})
    same(*out)
