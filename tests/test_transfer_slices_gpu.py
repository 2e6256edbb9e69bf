"""Particle uploads and downloads around the sizes where the host copies are
cut into slices: every value crosses unchanged."""
import numpy as np
import pytest

import CryoSPH as cs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,optional", [(1, True), (77_600, True), (77_700, False), (200_001, True), (700_003, False)])
def test_round_trip(cuda_device, n, optional, dtype):
    rng = np.random.default_rng(n)
    cfg = cs.SolverConfig()
    cfg.dx, cfg.normalize_initial_masses, cfg.phase_change = 0.01, False, False
    s = cs.Solver(cfg, cs.FluidProperties.water())
    f = lambda lo, hi, shape: rng.uniform(lo, hi, shape).astype(np.float32).astype(dtype)
    p = {"position": f(0, 1, (n, 3)), "mass": f(1e-4, 1e-3, n), "density": f(900, 1000, n),
         "temperature": f(290, 310, n)}
    phase = rng.choice(np.array([0, 2], np.uint8), n)
    extra = {}
    if optional:
        extra = {"velocity": f(-1, 1, (n, 3)), "normal": f(-1, 1, (n, 3)),
                 "flags": rng.integers(0, 2, n).astype(np.uint8)}
    s.set_particles(p["position"], p["mass"], p["density"], p["temperature"], phase, domain_lo=(0, 0, 0),
                    domain_hi=(1, 1, 1), **extra)
    q = s.particles()
    order = np.argsort(q["id"])
    assert np.array_equal(q["id"][order], np.arange(n))
    assert np.array_equal(q["phase"][order], phase)
    for k in ("position", "mass", "temperature"):
        assert np.array_equal(q[k][order], p[k].astype(np.float32)), k
    if optional:
        for k in ("velocity", "normal", "flags"):
            assert np.array_equal(q[k][order], extra[k].astype(q[k].dtype)), k


@pytest.mark.parametrize("n", [35_000, 36_500, 50_000, 72_000])
def test_one_slice_of_doubles(cuda_device, n):
    """Below one slice, doubles of more than 4 MiB are copied by several threads."""
    test_round_trip(cuda_device, n, True, np.float64)


@pytest.mark.parametrize("n", [1, 15, 17, 4099])
def test_phases_are_counted(cuda_device, n):
    """A tank is two-phase if any of its particles, the last included, is vapour."""
    cfg = cs.SolverConfig()
    cfg.dx = 0.01
    cfg.surface_tension = cs.SurfaceTensionModel.Akinci
    x = np.random.default_rng(n).uniform(0, 1, (n, 3))
    full = np.full(n, 1.0)
    for k in sorted({0, n // 2, n - 1}):
        phase = np.full(n, 2, np.uint8)
        s = cs.Solver(cfg, cs.FluidProperties.water())
        s.set_particles(x, full, full, full, phase, domain_lo=(0, 0, 0), domain_hi=(1, 1, 1))
        phase[k] = 1  # Akinci's model takes no vapour
        with pytest.raises(ValueError):
            s.set_particles(x, full, full, full, phase, domain_lo=(0, 0, 0), domain_hi=(1, 1, 1))
