"""A matrix that is not there is not multiplied by: builds that fail, builds anew
under the form in use, and profiles of a dense product that a context does not hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Vpl", "rake", "mu0", "sig", "a", "b", "L", "Vo", "damping")


def _model(ucg, nx, nz):
    from unicycle_b200 import configs
    c = configs.cfg2(nx=nx, nz=nz)
    sim = ucg.Simulation(c["mu"], c["lam"])
    sim.set_triangles(*c["mesh"]["tri"])
    sim.set_friction(*(c["friction"][k] for k in FIELDS))
    sim.set_tolerance(1.0e-8, 1.0e4)
    y = c["y0"].copy()
    y[6::7] += np.random.default_rng(nx).normal(0, 0.3, c["n_patch"])
    return sim, y


def _run(sim, y):
    sim.set_state(y, 0.0, 1.0e4)
    assert sim.run(1.0e30, 2) == 2
    return sim.get_state()[0]


@pytest.mark.parametrize("form", ["HMATRIX", "HMATRIX_SPLIT"])
def test_failed_build(ucg, form):
    """14,112 triangles in one leaf: its dense block (9.6 GB) exceeds the build scratch."""
    sim, y = _model(ucg, 84, 84)
    sim.build_hmatrix()
    sim.set_precision(getattr(ucg, "UCG_PREC_" + form))
    ref = _run(sim, y)
    sim.set_state(y, 0.0, 1.0e4)
    with pytest.raises(ucg.UcgError):
        sim.build_hmatrix(leaf=20000)
    for call in (lambda: sim.run(1.0e30, 1), lambda: sim.odefun(y), lambda: sim.set_state(y, 0.0, 1.0e4),
                 lambda: sim.step(0.0, y, 1.0e2), sim.hmatrix_info,
                 lambda: sim.set_precision(ucg.UCG_PREC_HMATRIX), sim.profile_traction):
        with pytest.raises(ucg.UcgError):
            call()
    sim.build_hmatrix()
    assert np.array_equal(_run(sim, y), ref)
    sim.close()


def test_build_anew_in_the_split_form(ucg):
    sim, y = _model(ucg, 20, 20)
    sim.build_hmatrix(leaf=24)
    sim.set_precision(ucg.UCG_PREC_HMATRIX_SPLIT)
    ref = _run(sim, y)
    sim.build_hmatrix(leaf=24)
    assert np.array_equal(_run(sim, y), ref)
    sim.close()


def test_profile_without_a_dense_matrix(ucg):
    sim, y = _model(ucg, 6, 6)
    sim.build_hmatrix(leaf=16)
    sim.set_precision(ucg.UCG_PREC_HMATRIX)
    _run(sim, y)
    with pytest.raises(ucg.UcgError):
        sim.profile_traction()
    sim.buildG()
    assert sim.profile_traction() > 0.0
    sim.close()
