"""A restored state chooses the shapes of the neighbour passes by its own
particles, not by those that were loaded before it."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import CryoSPH as cs

pytestmark = pytest.mark.gpu

DX = 0.004


def solver(layers, steps=2):
    """The lower layers of a box of 110 592 fluid particles, in the whole box's domain."""
    water = cs.FluidProperties.water()
    box = cs.BoxTank(48 * DX, 48 * DX, 48 * DX)
    fill = cs.FillSpec()
    fill.mode = cs.FillMode.Full
    p = cs.tank_particles(box, water, DX, fill)
    keep = (p["phase"] == 2) | (p["position"][:, 2] < p["position"][p["phase"] == 0][:, 2].min() + (layers - 0.5) * DX)
    q = {k: np.asarray(v)[keep] for k, v in p.items()}
    cfg = cs.SolverConfig()
    cfg.dx, cfg.surface_tension, cfg.thermal, cfg.phase_change = DX, cs.SurfaceTensionModel.NoTension, False, False
    cfg.velocity_scale, cfg.gravity = 1.0, (0.0, 0.0, -1.0)
    s = cs.Solver(cfg, water)
    lo, hi = cs.tank_domain(box, DX, 3)
    s.set_particles(q["position"], q["mass"], q["density"], q["temperature"], q["phase"], domain_lo=lo, domain_hi=hi,
                    normal=q["normal"], flags=q["flags"])
    if steps:
        s.run_steps(steps)
    return s


def kernels(s):
    """Shapes of the force pass over a few steps, in the replayed graph or not.
    A capture can miss the first kernels after it opens, hence several."""
    torch.zeros(1, device="cuda")
    names = set()
    for _ in range(4):
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            s.run_steps(3)
            s.diagnostics()
            torch.cuda.synchronize()
        names |= {e.key for e in prof.key_averages() if "k_forces_t" in e.key}
    if not names:
        pytest.skip("the profiler records no kernels here")
    return {"lanes" if "lanes::" in k else "threads" for k in names}


@pytest.mark.parametrize("graph", [False, True])
def test_restored_state_chooses_the_shapes(cuda_device, graph):
    small, large = solver(4), solver(48)
    for s in (small, large):
        s.set_graph_mode(graph)
        s.step()
    blobs = [s.save_state() for s in (small, large)]
    assert kernels(small) == {"lanes"} and kernels(large) == {"threads"}
    small.load_state(blobs[1])
    large.load_state(blobs[0])
    assert kernels(small) == {"threads"} and kernels(large) == {"lanes"}
    small.load_state(blobs[0])
    assert kernels(small) == {"lanes"}
    for s in (small, large):
        s.load_state(blobs[0])
        s.run_steps(3)
    a, b = small.particles(), large.particles()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def test_state_saved_before_the_first_step(cuda_device):
    """A state that has not been sorted is counted."""
    small, large = solver(4, 0), solver(48, 0)
    blob = large.save_state()
    small.load_state(blob)
    assert kernels(small) == {"threads"}
