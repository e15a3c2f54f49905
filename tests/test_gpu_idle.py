"""Attempts that have nothing to do.  ucg_run queues them in batches, so up to 31 run
behind the step that ends a run: each of their kernels has to see that at once.

A run that ends by its time after one step (a full batch is queued) against one that
ends by its count of steps (only that one is) gives the time of 31 idle attempts.  It
is launches alone, the same for every model: at 7,200 triangles, whose stages move
up to 1.2 GB, at most 1.5 times that of 148 rectangles (measured 1.2-1.3; the rest is
the first copy, which goes out before the kernel knows)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _seconds(sim, y0, t_end, steps):
    ts = []
    for _ in range(25):
        sim.set_state(y0, 0.0, 1.0e4)
        t = time.perf_counter()
        assert sim.run(t_end, steps) == 1
        ts.append(time.perf_counter() - t)
    return np.median(ts)


def _idle(sim, c):
    sim.set_tolerance(1.0e-8, 1.0e4)
    return _seconds(sim, c["y0"], 1.0, 1000) - _seconds(sim, c["y0"], 1.0e30, 1)


@pytest.fixture(scope="module")
def small(ucg):
    from unicycle_b200 import configs
    c = configs.tilt(configs.cfg1(nx=37, nz=4))
    sim = ucg.Simulation(c["mu"], c["lam"])
    configs.build(sim, c)
    t = _idle(sim, c)
    sim.close()
    return t


@pytest.mark.parametrize("form", ["fp64", "split_pair"])
def test_idle_attempts(ucg, small, form):
    from unicycle_b200 import configs
    c = configs.cfg2(nx=60, nz=60)
    sim = ucg.Simulation(c["mu"], c["lam"])
    configs.build(sim, c)
    sim.set_precision(form)
    t = _idle(sim, c)
    sim.close()
    print(f"31 idle attempts: {form} {1e6 * t:.0f} us, 148 rectangles {1e6 * small:.0f}")
    assert t <= 1.5 * small
