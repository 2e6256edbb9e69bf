"""The cell sort, the neighbour-list build and the neighbour passes at the
sizes where a change of launch shape or a remainder can go wrong.  Every
comparison is bit for bit: the shapes add the same terms in the same order."""
import numpy as np
import pytest

import CryoSPH as cs
import cryo_cabi as cabi

pytestmark = pytest.mark.gpu

LO, HI = (0.0, 0.0, 0.0), (0.4, 0.3, 0.2)


def cloud(n, seed, dense=0, outside=0):
    """n liquid particles: uniform in the domain, the first `dense` of them in
    one small clump, the last `outside` beyond the domain."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(LO, HI, (n, 3)).astype(np.float32)
    x[:dense] = (0.101 + 0.002 * rng.random((min(dense, n), 3))).astype(np.float32)
    if outside:
        x[-outside:] += np.float32(0.5)
    return {"x": x, "m": np.full(n, 1e-3, np.float32), "rho": np.full(n, 1000, np.float32),
            "T": np.full(n, 300, np.float32), "phase": np.zeros(n, np.uint8)}


def free_surface_config(dx, **kw):
    return cabi.py_config(dx=dx, gravity=(0, 0, -1.0), surface_tension=0, thermal=0, phase_change=0, density_mode=1,
                          velocity_scale=1.0, normalize_initial_masses=0, **kw)


@pytest.mark.parametrize("n,dense,outside", [(1, 0, 0), (2, 0, 1), (31, 0, 0), (33, 33, 0), (257, 200, 3), (2049, 0, 7),
                                             (6000, 700, 40)])
def test_cell_sort_is_the_stable_sort(cuda_device, n, dense, outside):
    g = cabi.Context(free_surface_config(0.01), cabi.py_fluid(cabi.FLUID_H2O))
    p = cloud(n, n, dense, outside)
    g.set_particles(p, LO, HI)
    for build in range(3):  # again on the sorted particles: the counters start from zero each time
        x = g.field("x")
        info = g.grid_info()
        inv = np.float32(1) / np.float32(info["cell"])
        c = np.floor((x - np.array(info["origin"], np.float32)) * inv)
        dims = np.array([info["nx"], info["ny"], info["nz"]])
        c = np.clip(c, 0, dims - 1).astype(np.int64)
        key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
        g.run_pass("grid_build")
        keys, perm, begin, end = g.grid_tables()
        order = np.argsort(key, kind="stable")
        assert np.array_equal(perm, order) and np.array_equal(keys, key[order])
        count = np.bincount(key, minlength=info["num_cells"])
        assert np.array_equal(end - begin, count)


def assert_stored_equal_scan(g, phase):
    sc, sl = g.neighbor_lists(stored=True)
    gc, gl = g.neighbor_lists()
    owner = np.repeat(np.arange(len(gc)), gc)
    keep = (phase[owner] != 2) | (phase[gl] <= 1)  # a wall's stored list holds its fluid neighbours
    assert np.array_equal(sc, np.bincount(owner[keep], minlength=len(gc)))
    assert np.array_equal(sl, gl[keep])


@pytest.mark.parametrize("n", [1, 3, 7, 9, 63, 64, 65, 255, 1025, 4099])
def test_lists_of_random_clouds(cuda_device, n):
    g = cabi.Context(free_surface_config(0.012), cabi.py_fluid(cabi.FLUID_H2O))
    p = cloud(n, 7 * n)
    p["phase"][::5] = 2  # some walls among them
    g.set_particles(p, LO, HI)
    g.run_pass("grid_build")
    assert_stored_equal_scan(g, g.field("phase"))


def big_tank():
    water = cs.FluidProperties.water()
    fill = cs.FillSpec()
    fill.fill_fraction = 0.55
    return water, cs.tank_particles(cs.BoxTank(0.27, 0.25, 0.26), water, 0.004, fill), cs.tank_domain(
        cs.BoxTank(0.27, 0.25, 0.26), 0.004, 3)


def test_lists_of_a_large_tank(cuda_device):
    """More particles than the list build shares lanes over, in the one-thread shape."""
    _, p, (lo, hi) = big_tank()
    n = len(p["mass"])
    assert n > 300_000
    g = cabi.Context(cabi.py_config(dx=0.004, thermo_mode=1), cabi.py_fluid(cabi.FLUID_H2O))
    g.set_particles({"x": p["position"], "m": p["mass"], "rho": p["density"], "T": p["temperature"],
                     "phase": p["phase"], "nrm": p["normal"]}, lo, hi)
    g.run_pass("grid_build")
    assert_stored_equal_scan(g, g.field("phase"))


@pytest.mark.parametrize("phase_change", [0, 1])
def test_more_neighbours_than_the_lists_hold(cuda_device, phase_change):
    """Particles with over 128 neighbours search the cells instead; a tank in
    which some do equals one stepped without lists."""
    p = cloud(900, 3, dense=0)
    p["x"][:400] = np.random.default_rng(1).uniform((0.1, 0.1, 0.1), (0.13, 0.13, 0.13), (400, 3)).astype(np.float32)
    p["phase"][100:160] = 1
    p["phase"][160:220] = 2
    p["T"][:100] = 380.0
    cfg = cabi.py_config(dx=0.012, gravity=(0, 0, -1.0), velocity_scale=1.0, thermo_mode=1, heater_power=3.0,
                         phase_change=phase_change, fixed_dt=1e-6)
    out = []
    for lists in (1, 0):
        g = cabi.Context(cfg, cabi.py_fluid(cabi.FLUID_H2O))
        g.set_neighbor_mode(lists)
        g.set_particles(p, LO, HI)
        g.step(3)
        if lists:
            assert g.neighbor_lists()[0].max() > 128
        out.append({f: g.field(f) for f in ("x", "v", "rho", "T", "m", "p", "a", "sigma", "nrm", "kappa", "fw", "mw")})
    for f in out[0]:
        assert np.array_equal(out[0][f].view(np.uint32), out[1][f].view(np.uint32)), f


def small_tanks():
    """Two-phase and free-surface tanks over the options the passes branch on."""
    ln2, h2o = cs.FluidProperties.liquid_nitrogen, cs.FluidProperties.water

    def make(geo, fluid, fill, seed, **kw):
        cfg = cs.SolverConfig()
        cfg.dx = 0.004
        for k, v in kw.items():
            cur = getattr(cfg, k)
            setattr(cfg, k, type(cur)(v) if hasattr(cur, "value") else v)
        s = cs.Solver(cfg, fluid)
        s.build_tank(geo, fill)
        s.jitter_fluid(0.0002, seed)
        return s

    def fill(fraction, dT=0.0, vapour=True):
        f = cs.FillSpec()
        f.fill_fraction = fraction
        f.include_vapor = vapour
        if dT:
            f.T_liquid = ln2().T_sat + dT
        return f

    return [
        lambda: make(cs.BoxTank(0.03, 0.03, 0.03), ln2(), fill(0.5, 3.0), 1, gravity=(0.1, 0, -0.5)),
        lambda: make(cs.CylinderTank(0.03, 0.06), ln2(), fill(0.4, 2.0), 2, heater_power=20.0, thermo_mode=1,
                     wetting_model=2),
        lambda: make(cs.SphereTank(0.03), ln2(), fill(0.6), 3, csf_balanced=True, sps_turbulence=True,
                     transport_stress=True, wall_thermal_bc=1, thermo_mode=1),
        lambda: make(cs.BoxTank(0.04, 0.03, 0.03), h2o(), fill(0.5, vapour=False), 4, surface_tension=2, thermal=False,
                     phase_change=False, velocity_scale=0.5, gravity=(0, 0, -1.0)),
        lambda: make(cs.BoxTank(0.04, 0.03, 0.03), h2o(), fill(0.5, vapour=False), 5, surface_tension=0, thermal=False,
                     phase_change=False, density_mode=1, velocity_scale=0.5, gravity=(0, 0, -1.0), no_slip=False),
    ]


def test_lanes_and_threads_give_the_same_bits(cuda_device):
    """A small tank alone steps with lanes sharing its particles; beside a
    tank that fills the chip it steps with a thread per particle."""
    water, p, (lo, hi) = big_tank()
    cfg = cs.SolverConfig()
    cfg.dx = 0.004
    filler = cs.Solver(cfg, water)
    filler.set_particles(p["position"], p["mass"], p["density"], p["temperature"], p["phase"], domain_lo=lo,
                         domain_hi=hi, normal=p["normal"], flags=p["flags"])
    crowd, alone = cs.Ensemble(0), [make() for make in small_tanks()]
    beside = [make() for make in small_tanks()]
    crowd.add(filler)
    for s in beside:
        crowd.add(s)
    crowd.run_steps(6)
    for a, b in zip(alone, beside):
        a.run_steps(6)
        pa, pb = a.particles(), b.particles()
        for k in pa:
            assert np.array_equal(np.asarray(pa[k]).view(np.uint8), np.asarray(pb[k]).view(np.uint8)), k
        assert a.diagnostics().as_dict() == b.diagnostics().as_dict()


# (options, what takes the force pass off the instance with the rarer options
# compiled out without changing a value, arithmetics that have such an instance)
OTHER_ROUTE = [
    (dict(surface_tension=0, thermal=0, density_mode=0), dict(csf_balanced=1), (0, 1)),
    (dict(surface_tension=0, thermal=0, density_mode=1, no_slip=0), dict(csf_balanced=1), (0, 1)),
    (dict(surface_tension=0, thermal=1, density_mode=0), dict(csf_balanced=1), (0,)),
    (dict(surface_tension=0, thermal=1, density_mode=1), dict(csf_balanced=1), (0,)),
    (dict(surface_tension=1, thermal=0, density_mode=0), dict(wall_thermal_bc=1), (0, 1)),
    (dict(surface_tension=1, thermal=0, density_mode=1), dict(wall_thermal_bc=1), (0,)),
    (dict(surface_tension=1, thermal=1, density_mode=0), dict(sps_turbulence=1, smagorinsky_cs=0.0), (0,)),
    (dict(surface_tension=1, thermal=1, density_mode=1), dict(sps_turbulence=1, smagorinsky_cs=0.0), (0,)),
    # all temperatures equal: an isothermal wall exchanges nothing
    (dict(surface_tension=1, thermal=1, density_mode=0, T=300.0), dict(wall_thermal_bc=1), (0, 1)),
]


@pytest.mark.parametrize("base,other,arithmetics", OTHER_ROUTE)
def test_force_pass_without_the_rarer_options(cuda_device, base, other, arithmetics):
    _, p, (lo, hi) = big_tank()
    base = dict(base)
    T = np.full(len(p["mass"]), base.pop("T"), np.float32) if "T" in base else p["temperature"]
    x = p["position"] + np.random.default_rng(5).uniform(-2e-4, 2e-4, p["position"].shape).astype(np.float32)
    for arithmetic in arithmetics:
        out = []
        for extra in ({}, other):
            g = cabi.Context(cabi.py_config(dx=0.004, gravity=(0, 0, -1.0), phase_change=0, thermo_mode=1,
                                            transport_velocity=1, **base, **extra), cabi.py_fluid(cabi.FLUID_H2O))
            g.set_field_arithmetic(arithmetic)
            g.set_particles({"x": x, "m": p["mass"], "rho": p["density"], "T": T, "phase": p["phase"],
                             "nrm": p["normal"]}, lo, hi)
            g.step(2)
            out.append({f: g.field(f) for f in ("x", "v", "rho", "T", "a", "ab", "drho", "dTdt", "fw", "mw")})
        for f in out[0]:
            assert np.array_equal(out[0][f].view(np.uint32), out[1][f].view(np.uint32)), (arithmetic, f)


@pytest.mark.parametrize("np_", [1, 3, 4, 5, 1024, 1025])
def test_probes_by_warps(cuda_device, np_):
    """Any number of points gives each point's own value, that of the sum over
    the liquid (a term is within 16 ulp, at most ~100 of them are added)."""
    cfg = free_surface_config(0.02)
    g = cabi.Context(cfg, cabi.py_fluid(cabi.FLUID_H2O))
    g.set_particles(cloud(6000, 11), LO, HI)
    g.step(1)
    pts = np.random.default_rng(np_).uniform((-0.05, -0.05, -0.05), (0.45, 0.35, 0.25), (np_, 3)).astype(np.float32)
    p = np.asarray(g.probe_pressure(pts))
    for k in range(0, np_, max(1, np_ // 5)):
        one = np.asarray(g.probe_pressure(pts[k:k + 1]))
        assert np.array_equal(one.view(np.uint32), p[k:k + 1].view(np.uint32)) or (np.isnan(one[0]) and np.isnan(p[k]))
        h = 0.02 * 1.3
        q = np.linalg.norm(g.field("x").astype(np.float64) - pts[k].astype(np.float64), axis=1) / h
        w = np.where(q < 2, (1 - q / 2) ** 4 * (2 * q + 1), 0.0) * g.field("m") / g.field("rho")
        if w.sum() > 1e-3 * (1e-3 / 1000):
            term = w * g.field("p")
            assert abs(one[0] - term.sum() / w.sum()) <= 2e-4 * np.abs(term).sum() / w.sum()


@pytest.mark.parametrize("arithmetic", [0, 1])
@pytest.mark.parametrize("np_", [32768, 32769, 40001])
def test_probes_of_many_points(cuda_device, np_, arithmetic):
    """Above 32 768 points each has a thread instead of a warp: the same bits."""
    g = cabi.Context(free_surface_config(0.02), cabi.py_fluid(cabi.FLUID_H2O))
    g.set_field_arithmetic(arithmetic)
    g.set_particles(cloud(6000, 11), LO, HI)
    g.step(1)
    pts = np.random.default_rng(np_).uniform((-0.05, -0.05, -0.05), (0.45, 0.35, 0.25), (np_, 3)).astype(np.float32)
    p = np.asarray(g.probe_pressure(pts))
    parts = np.concatenate([np.asarray(g.probe_pressure(q)) for q in np.array_split(pts, 9)])
    assert np.array_equal(np.isnan(p), np.isnan(parts)) and 0 < np.isnan(p).sum() < np_
    assert np.array_equal(p[~np.isnan(p)].view(np.uint32), parts[~np.isnan(p)].view(np.uint32))
