"""Right-hand sides with infinite operands, against the oracle's divisions: a state
variable so small that exp(-psi ln 10) overflows (the rates are infinite, not NaN),
velocities that underflow, and an infinite weakening distance L (no state evolution by
slip: everything stays finite, and a step is taken).

Tolerance: 1e-12 of the component's largest finite entry, as the finite right-hand
sides elsewhere; infinities and NaN where the oracle has them."""
import numpy as np
import pytest

from test_gpu_attempts import _compare, _reference_step

pytestmark = pytest.mark.gpu

FIELDS = ("Vpl", "rake", "mu0", "sig", "a", "b", "L", "Vo", "damping")


def _model(ucg, oracle_lib, **changed):
    from unicycle_b200 import configs
    n = 9
    c = configs.tilt(configs.cfg1(nx=n, nz=1, seed=n))
    fr = {k: np.array(c["friction"][k], float) * np.ones(n) for k in FIELDS}
    for k, v in changed.items():
        fr[k][3] = v
    sim = ucg.Simulation(c["mu"], c["lam"])
    configs.build(sim, c)
    sim.set_friction(*(fr[k] for k in FIELDS))
    y = c["y0"].copy()
    y[6::7] += np.random.default_rng(n).normal(0, 0.3, n)
    return sim, oracle_lib.Model(sim.copy_G(), fr), y


@pytest.mark.parametrize("changed,entry,value", [({}, 5, -400.0), ({}, 5, -np.inf), ({}, 5, np.inf), ({}, 6, -400.0),
                                                 ({"b": 0.0}, 5, -400.0), ({"L": np.inf}, 5, None),
                                                 ({"L": np.inf}, 5, 2.0)])
def test_rates(ucg, oracle_lib, changed, entry, value):
    sim, ref, y = _model(ucg, oracle_lib, **changed)
    if value is not None:
        y[7 * 3 + entry] = value
    d = sim.odefun(y)[0]
    r = ref.odefun(y)[0]
    sim.close()
    for q in range(7):
        a, b = d[q::7], r[q::7]
        ok = np.isfinite(b)
        assert np.array_equal(a[~ok], b[~ok], equal_nan=True)
        assert np.max(np.abs(a[ok] - b[ok])) <= 1e-12 * np.max(np.abs(b[ok]))


def test_step_without_state_evolution(ucg, oracle_lib):
    sim, _, y = _model(ucg, oracle_lib, L=np.inf)
    ref, hd, _, nrej = _reference_step(lambda x: sim.odefun(x)[0], y, 1.0e2, 1.0e-6)
    sim.set_tolerance(1.0e-6)
    t, yn, _, _, dd, rej = sim.step(0.0, y, 1.0e2)
    sim.close()
    assert rej == nrej and abs(dd - hd) <= 1e-6 * hd
    _compare(y, yn, ref, 9, 0, 1e-6)
