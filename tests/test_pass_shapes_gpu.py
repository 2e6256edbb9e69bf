"""The cell sort and the neighbour-list build at the sizes where a change of
launch shape or a remainder can go wrong, bit for bit."""
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
