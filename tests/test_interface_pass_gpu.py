"""The interface pass leaves out particles with no wall and none of the other
phase in the cells around them, as the last sort found them.  Outside a step
the phases may have been set since: the pass then has to take them as they are."""
import numpy as np
import pytest

import CryoSPH as cs
import cryo_cabi as cabi

pytestmark = pytest.mark.gpu

DX = 0.004
FIELDS = ("nrm", "alpha", "wall_w", "heat_w", "vw", "ns")


def tank(arithmetic, lists, **kw):
    """A two-phase box of 8 000 fluid particles; its bulk is far from walls and interface."""
    fluid = cs.FluidProperties.liquid_nitrogen()
    geometry = cs.BoxTank(20 * DX, 20 * DX, 20 * DX)
    fill = cs.FillSpec()
    fill.fill_fraction = 0.5
    p = cs.tank_particles(geometry, fluid, DX, fill)
    lo, hi = cs.tank_domain(geometry, DX, 3)
    x = p["position"] + np.random.default_rng(3).uniform(-3e-4, 3e-4, p["position"].shape).astype(np.float32)
    g = cabi.Context(cabi.py_config(dx=DX, gravity=(0, 0, -0.01), thermo_mode=1, **kw), cabi.py_fluid(cabi.FLUID_LN2))
    g.set_neighbor_mode(lists)
    g.set_field_arithmetic(arithmetic)
    g.set_particles({"x": x, "m": p["mass"], "rho": p["density"], "T": p["temperature"], "phase": p["phase"],
                     "nrm": p["normal"], "flags": p["flags"]}, lo, hi)
    return g


def turn_a_blob_over(g):
    """The other phase for the fluid particles of two blobs inside the liquid and the vapour."""
    x, phase = g.field("x"), g.field("phase")
    fluid = phase <= 1
    mid = 0.5 * (x[fluid].min(0) + x[fluid].max(0))
    for z in (-0.25, 0.25):
        blob = fluid & (np.linalg.norm(x - (mid + np.array([0, 0, z * 20 * DX])), axis=1) < 2 * DX)
        assert blob.sum() > 10
        phase[blob] = 1 - phase[blob]
    g.set_field("phase", phase)


def same(a, b):
    for f in a:
        assert np.array_equal(a[f].view(np.uint32), b[f].view(np.uint32)), f


@pytest.mark.parametrize("arithmetic", [0, 1])
def test_interface_pass_takes_the_phases_as_they_are(cuda_device, arithmetic):
    out = []
    for lists in (1, 0):
        g = tank(arithmetic, lists)
        for name in ("grid_build", "density", "eos", "wall_boundary"):
            g.run_pass(name)
        turn_a_blob_over(g)
        g.run_pass("interface")
        out.append({f: g.field(f) for f in FIELDS})
    same(*out)


@pytest.mark.parametrize("arithmetic", [0, 1])
def test_rates_after_relax_take_the_phases_as_they_are(cuda_device, arithmetic):
    """relax() closes with an evaluation of the rates that no sort precedes:
    it leaves the interface fields an operator pass gives, and in the exact
    arithmetic the rates found without lists."""
    out = []
    for lists in (1, 0):
        g = tank(arithmetic, lists)
        g.step(1)
        turn_a_blob_over(g)
        g.relax(0.0)
        out.append({f: g.field(f) for f in FIELDS + ("a", "kappa", "p")})
        left = {f: g.field(f) for f in FIELDS}
        g.run_pass("interface")
        same(left, {f: g.field(f) for f in FIELDS})
    if arithmetic == 0:
        same(*out)
