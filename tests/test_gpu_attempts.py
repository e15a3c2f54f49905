"""Whole attempts at the sizes where the fused stage kernels can go wrong: one
element, fewer elements than CTAs, one more or less than the 148 of a full
grid, patches beside volumes, hierarchical leaves that are not a multiple of the
8 patches a CTA takes, ensembles around the 32- and 128-element blocks; accepted
at once, and after rejections, which repeat from the same first stage.

The reference is the Cash-Karp attempt and the RKQSm decision
(fortran/3d/src/ode45.f90:51-200) written out here, over right-hand sides f(y)
that the other tests pin to the oracle.

Tolerances, on the change of the state over the step, per group of components
(slip, traction, theta, V; strain, stress) against the group's largest change.
FP64 and hierarchical FP64: both sides round f to about 1e-13 of its terms; the
error estimate is the 1e-6 part of it at the tolerance used, so the step that a
rejection chooses agrees to 1e-13 / 1e-6 = 1e-7, and with it every change: 1e-6.
Split forms: products to 3e-7 (pair) or, in the increments, 2^-11 (bf16) of |K||v|,
some 10 times the sum's size; the estimate is the 1e-3 part of the rates, so the step
agrees to 0.2 * 10 * 2^-11 / 1: 2e-2 covers both.  The ensembles' contraction
(1e-5 of |K||v|): the same 2e-2.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

B = [[], [0.2], [3 / 40, 9 / 40], [0.3, -0.9, 1.2], [-11 / 54, 2.5, -70 / 27, 35 / 27],
     [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]]
C = np.array([37 / 378, 0, 250 / 621, 125 / 594, 0, 512 / 1771])
D = C - np.array([2825 / 27648, 0, 18575 / 48384, 13525 / 55296, 277 / 14336, 0.25])


def _reference_step(f, y, h, eps, hmax=1.7976931348623158e308):
    k1 = f(y)
    yscal = np.abs(y) + np.abs(h * k1) + 1e-30
    nrej = 0
    while True:
        k = [k1]
        for s in range(1, 6):
            k.append(f(y + h * sum(b * kk for b, kk in zip(B[s], k))))
        k = np.array(k)
        err = np.max(np.abs(h * (D @ k)) / yscal) / eps
        if err <= 1.0:
            break
        h *= 0.7 * err ** -0.15
        nrej += 1
        assert nrej < 50
    hn = 0.7 * h * err ** -0.2 if err > 1.89e-4 else 10.0 * h
    return y + h * (C @ k), h, min(hn, hmax), nrej


def _groups(np_, nv):
    p = np.arange(7 * np_).reshape(-1, 7)
    v = 7 * np_ + np.arange(12 * nv).reshape(-1, 12)
    return [g.ravel() for g in (p[:, :2], p[:, 2:5], p[:, 5:6], p[:, 6:7], v[:, :6], v[:, 6:]) if g.size]


def _compare(y0, y, ref, np_, nv, tol):
    for g in _groups(np_, nv):
        d, r = (y - y0)[g], (ref - y0)[g]
        lim = tol * np.abs(r).max() + 4.0 * np.spacing(np.abs(y0[g]).max())
        assert np.abs(d - r).max() <= lim, (g[:3], np.abs(d - r).max(), lim)


def _patches(ucg, n, leaf=None):
    from unicycle_b200 import configs
    c = configs.tilt(configs.cfg1(nx=n, nz=1, seed=n))
    y0 = c["y0"].copy()
    y0[6::7] += np.random.default_rng(n).normal(0, 0.3, n)
    sim = ucg.Simulation(c["mu"], c["lam"])
    configs.build(sim, c)
    if leaf:
        sim.build_hmatrix(eta=2.0, eps=1e-6, leaf=leaf)
        sim.set_precision(ucg.UCG_PREC_HMATRIX)
    return sim, y0


@pytest.mark.parametrize("h", [1.0e2, 2.0e6])
@pytest.mark.parametrize("n,leaf", [(1, None), (3, None), (147, None), (148, None), (149, None), (593, None),
                                    (33, 5), (150, 12), (150, 33)])
def test_step_of_patches(ucg, n, leaf, h):
    sim, y0 = _patches(ucg, n, leaf)
    eps = 1.0e-6
    ref, hd, hn, nrej = _reference_step(lambda y: sim.odefun(y)[0], y0, h, eps)
    sim.set_tolerance(eps)
    t, y, dydt, dn, dd, rej = sim.step(0.0, y0, h)
    assert rej == nrej and (n < 100 or (nrej > 0) == (h > 1e3))
    assert np.array_equal(dydt, sim.odefun(y0)[0])
    assert abs(dd - hd) <= 1e-6 * hd and t == dd and abs(dn - hn) <= 1e-6 * hn
    _compare(y0, y, ref, n, 0, 1e-6)
    sim.close()


@pytest.mark.parametrize("h", [1.0e2, 2.0e6])
@pytest.mark.parametrize("nxf,nzf,nxv,nyv,nzv", [(1, 1, 1, 1, 1), (3, 1, 2, 1, 1), (60, 1, 11, 4, 2), (9, 5, 7, 5, 3)])
def test_step_of_patches_and_volumes(ucg, nxf, nzf, nxv, nyv, nzv, h):
    from unicycle_b200 import configs
    # tilted, and the volumes off the fault's plane of symmetry: no component is
    # rounding residue, on which the relative error norm would act
    c = configs.cfg3(nxf=nxf, nzf=nzf, nxv=nxv, nyv=nyv, nzv=nzv)
    c["mesh"]["vol"][0][:, 0] += 317.0
    c["y0"] = c["y0"][:7 * c["n_patch"]]
    c = configs.tilt(c)
    c["y0"] = np.concatenate([c["y0"], np.zeros(12 * c["n_vol"])])
    sim = ucg.Simulation(c["mu"], c["lam"], driver="viscouscycles")
    configs.build_coupled(sim, c)
    y0 = configs.coseismic_preload(sim.copy_G(), c)
    eps = 1.0e-6
    ref, hd, hn, nrej = _reference_step(lambda y: sim.odefun(y)[0], y0, h, eps)
    sim.set_tolerance(eps)
    t, y, dydt, dn, dd, rej = sim.step(0.0, y0, h)
    assert rej == nrej
    assert abs(dd - hd) <= 1e-6 * hd and t == dd and abs(dn - hn) <= 1e-6 * hn
    _compare(y0, y, ref, c["n_patch"], c["n_vol"], 1e-6)
    sim.close()


@pytest.mark.parametrize("h", [1.0e2, 1.0e6])
@pytest.mark.parametrize("form", ["SPLIT_PAIR", "SPLIT_BF16"])
@pytest.mark.parametrize("n", [1, 7, 149, 8 * 148 + 1])
def test_step_of_split_forms(ucg, n, form, h):
    sim, y0 = _patches(ucg, n)
    eps = 1.0e-3
    ref, hd, hn, nrej = _reference_step(lambda y: sim.odefun(y)[0], y0, h, eps)
    sim.set_precision(getattr(ucg, "UCG_PREC_" + form))
    sim.set_tolerance(eps)
    t, y, _, dn, dd, rej = sim.step(0.0, y0, h)
    assert rej == nrej
    assert abs(dd - hd) <= 2e-2 * hd
    _compare(y0, y, ref, n, 0, 2e-2)
    sim.close()


@pytest.mark.parametrize("h", [1.0e2, 1.0e6])
@pytest.mark.parametrize("n,ninst,leaf", [(1, 1, None), (31, 3, None), (33, 33, None), (128, 3, None), (129, 65, None),
                                          (130, 3, 12), (260, 33, 33)])
def test_ensemble_step(ucg, n, ninst, leaf, h):
    """Every instance with its own friction and state, to its first accepted step,
    beside instances that go on or repeat."""
    from unicycle_b200 import configs
    sim, _ = _patches(ucg, n, leaf)
    c = configs.tilt(configs.cfg1(nx=n, nz=1, seed=n))
    fr = c["friction"]
    eps = 1.0e-3
    rng = np.random.default_rng(n + ninst)
    ens = ucg.Ensemble()
    ens.add_geometry(sim, ninst)
    ens.set_tolerance(eps)
    y0, par = [], []
    for i in range(ninst):
        y = c["y0"].copy()
        y[6::7] += rng.normal(0, 0.3, n)
        L = fr["L"] * (1.0 + i)
        ens.set_friction(0, i, fr["Vpl"], fr["rake"], fr["mu0"], fr["sig"], fr["a"], fr["b"], L, fr["Vo"],
                         fr["damping"])
        y0.append(y)
        par.append(L)
    y0 = np.array(y0)
    ens.set_states(0, y0, 0.0, h)
    done = {}
    for _ in range(60):
        ens.run(1.0e30, 1)
        y, t, dn, acc, rej, st = ens.get_states(0)
        assert not st.any()
        for i in range(ninst):
            if acc[i] >= 1 and i not in done:
                done[i] = (y[i].copy(), t[i], rej[i])
        if len(done) == ninst:
            break
    assert len(done) == ninst
    for i in sorted({0, ninst // 2, ninst - 1}):
        sim.set_friction(fr["Vpl"], fr["rake"], fr["mu0"], fr["sig"], fr["a"], fr["b"], par[i], fr["Vo"], fr["damping"])
        ref, hd, hn, nrej = _reference_step(lambda z: sim.odefun(z)[0], y0[i], h, eps)
        yi, ti, ri = done[i]
        assert ri == nrej and abs(ti - hd) <= 2e-2 * hd, (i, ri, nrej, ti, hd)
        _compare(y0[i], yi, ref, n, 0, 2e-2)
    ens.close()
    sim.close()
