"""Attempts over which the rates change, so that every stage's weights and the error
vector count: the step is chosen where the last stage's rates differ from the first's
by a fifth to all of them, the accuracy so that the error is 0.8 of it (accepted at
once, and the next step follows from the error) or 50 times (repeated).

Single instances take f(y) from the same form's odefun, whose product is the same
matrix: the stages' increments over stage 1 are then the same sum in another order,
and both sides agree to 1e-13 of its terms, the step that a rejection chooses, the
next step and the changes to 1e-6 with margin.  Ensembles multiply to 1e-5 of |K||v|:
ten times that, over the sums' own size, of the changes.  (Their next step follows
from the one component of the largest relative error, of whose traction that error
may be any part.)
"""
import numpy as np
import pytest

from test_gpu_attempts import B, D, _compare, _patches, _reference_step

pytestmark = pytest.mark.gpu

LN10 = np.log(10.0)


def _curved(f, y, h=8.0e6):
    """A step with the rates' change in that range, and its error at unit accuracy."""
    k1 = f(y)
    while True:
        with np.errstate(all="ignore"):
            k = [k1]
            for s in range(1, 6):
                k.append(f(y + h * sum(b * kk for b, kk in zip(B[s], k))))
        k = np.array(k)
        if np.all(np.isfinite(k)):
            d = np.abs(k[5] - k[0])[6::7].max() / np.abs(k[0])[6::7].max()
            if d <= 1.0:
                break
        h /= 1.3
    assert d >= 0.2, d
    return h, np.max(np.abs(h * (D @ k)) / (np.abs(y) + np.abs(h * k1) + 1e-30))


@pytest.mark.parametrize("part", [0.8, 50.0])
@pytest.mark.parametrize("n,leaf,form", [(149, None, "FP64"), (7, None, "SPLIT_PAIR"), (8 * 148 + 1, None, "SPLIT_PAIR"),
                                         (33, 5, "HMATRIX"), (33, 5, "HMATRIX_SPLIT"), (150, 12, "HMATRIX_SPLIT"),
                                         (150, 33, "HMATRIX_SPLIT"), (150, 100, "HMATRIX_SPLIT")])
def test_step(ucg, n, leaf, form, part):
    sim, y0 = _patches(ucg, n, leaf)
    sim.set_precision(getattr(ucg, "UCG_PREC_" + form))

    def f(y):
        try:
            return sim.odefun(y)[0]
        except ucg.UcgError:         # a stage too far out
            return np.full(len(y), np.nan)
    h, err = _curved(f, y0)
    eps = err / part
    ref, hd, hn, nrej = _reference_step(f, y0, h, eps)
    assert (nrej > 0) == (part > 1.0)
    sim.set_tolerance(eps)
    t, y, _, dn, dd, rej = sim.step(0.0, y0, h)
    sim.close()
    assert rej == nrej
    assert abs(dd - hd) <= 1e-6 * hd and abs(dn - hn) <= 1e-6 * hn
    _compare(y0, y, ref, n, 0, 1e-6)


def _rates(K, fr):
    """f(y) of the patches (ratestate.f90:667-776), and the largest |K||v| / |K v|."""
    absK, far = np.abs(K), [0.0]

    def f(y):
        s = y.reshape(-1, 7)
        vel, rake = 10.0 ** s[:, 6], np.arctan2(s[:, 3], s[:, 2])
        c, d = np.cos(rake), np.sin(rake)
        v = np.stack([vel * c - fr["Vpl"] * np.cos(fr["rake"]), vel * d - fr["Vpl"] * np.sin(fr["rake"])], 1).ravel()
        t = K @ v
        far[0] = max(far[0], (absK @ np.abs(v)).max() / np.abs(t).max())
        t = t.reshape(-1, 3)
        dth = (10.0 ** -s[:, 5] - vel / fr["L"]) / LN10
        dv = (t[:, 0] * c + t[:, 1] * d - fr["b"] * fr["sig"] * dth * LN10) / (fr["a"] * fr["sig"] +
                                                                             fr["damping"] * vel) / LN10
        corr = fr["damping"] * vel * dv * LN10
        return np.stack([vel * c, vel * d, t[:, 0] - corr * c, t[:, 1] - corr * d, t[:, 2], dth, dv], 1).ravel()
    return f, far


@pytest.mark.parametrize("n,ninst,leaf", [(31, 3, None), (129, 33, None), (130, 3, 12), (260, 33, 33)])
def test_ensemble_step(ucg, n, ninst, leaf):
    from unicycle_b200 import configs
    sim, _ = _patches(ucg, n, leaf)
    K = sim.copy_G()
    c = configs.tilt(configs.cfg1(nx=n, nz=1, seed=n))
    keys = ("Vpl", "rake", "mu0", "sig", "a", "b", "L", "Vo", "damping")
    base = {k: np.array(c["friction"][k], float) * np.ones(n) for k in keys}
    rng = np.random.default_rng(n + ninst)
    fr, y0 = [], []
    for i in range(ninst):
        fr.append(base | {"L": base["L"] * (1.0 + 0.1 * i)})
        y0.append(c["y0"].copy())
        y0[i][6::7] += rng.normal(0, 0.3, n)
    h, err = _curved(_rates(K, fr[0])[0], y0[0])
    ens = ucg.Ensemble()
    ens.add_geometry(sim, ninst)
    ens.set_tolerance(1.0e3 * err)       # accepted at once, whatever an instance's error
    for i in range(ninst):
        ens.set_friction(0, i, *(fr[i][k] for k in keys))
    ens.set_states(0, np.array(y0), 0.0, h)
    ens.run(1.0e30, 1)
    y, t, dn, acc, rej, st = ens.get_states(0)
    ens.close()
    sim.close()
    assert not st.any() and np.all(acc == 1) and np.all(rej == 0) and np.all(t == h)
    for i in range(ninst):
        f, far = _rates(K, fr[i])
        ref, _, _, _ = _reference_step(f, y0[i], h, 1.0e3 * err)
        assert far[0] < 100.0
        _compare(y0[i], y[i], ref, n, 0, 10.0 * 1e-5 * far[0])
