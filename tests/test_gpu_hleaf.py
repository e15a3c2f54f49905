"""Hierarchical matrices with leaves of more patches than a CTA of the row kernel has
threads for (42): the product, and runs on it, at the first size beyond, leaves that
do not divide evenly, one leaf that is the whole model (a single dense block), and
more rows in it than a block of threads can have.

Tolerances.  Product: every low-rank block is checked to 10 eps of its own product
at the build (dense ones are exact), so |H x - K x| <= 10 eps sum |K| |x| per row.
A step over the same form's f(y): both sides round f to 1e-13 (FP64), so the
change agrees to 1e-6 with margin; the split form multiplies the stages' increments
by values rounded to 2^-24, some 10 times that of the sum: 1e-5."""
import numpy as np
import pytest

from test_gpu_attempts import _compare, _reference_step

pytestmark = pytest.mark.gpu

EPS = 1.0e-6


@pytest.mark.parametrize("nx,nz,leaf", [(9, 5, 44), (9, 5, 45), (11, 9, 64), (11, 9, 99), (16, 16, 300), (25, 8, 4000)])
def test_wide_leaves(ucg, nx, nz, leaf):
    from unicycle_b200 import configs
    c = configs.cfg2(nx=nx, nz=nz)
    n = c["n_patch"]
    sim = ucg.Simulation(c["mu"], c["lam"])
    configs.build(sim, c)
    K = sim.copy_G()
    sim.build_hmatrix(eps=EPS, leaf=leaf)
    x = np.random.default_rng(leaf).standard_normal(K.shape[1])
    assert np.all(np.abs(sim.hmatrix_matvec(x) - K @ x) <= 10 * EPS * (np.abs(K) @ np.abs(x)))
    y0, h = c["y0"].copy(), 1.0e2
    y0[6::7] += np.random.default_rng(n).normal(0, 0.3, n)
    for form, tol in ((ucg.UCG_PREC_HMATRIX, 1e-6), (ucg.UCG_PREC_HMATRIX_SPLIT, 1e-5)):
        sim.set_precision(form)
        ref, _, _, nrej = _reference_step(lambda y: sim.odefun(y)[0], y0, h, 1.0e-6)
        assert nrej == 0
        sim.set_tolerance(1.0e-6)
        sim.set_state(y0, 0.0, h)
        assert sim.run(1.0e30, 1) == 1
        _compare(y0, sim.get_state()[0], ref, n, 0, tol)
    sim.close()
