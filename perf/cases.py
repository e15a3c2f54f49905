"""Measured workloads of the 3-D quasi-dynamic solver.

Each case is one pass that a user's program makes through the public entry
points of `unicycle_b200`: assembling the Green's functions (`buildG`) and
taking the first right-hand side, compressing them (`build_hmatrix`), marching
a model (`step` with host arrays, `set_state` / `run` / `get_state` on the
device, every storage form of K), and marching an ensemble of parameter sets.
Meshes and frictional properties are the ones of `unicycle_b200.configs`.

The marching cases limit the step (`set_tolerance(epsilon, maximum_step)`, the
reference's --maximum-step) below what the error control would take, so that a
pass always makes the same accepted steps.

`exact` restates the same passes in 64 bits with torch alone: the Nikkhoo-Walter
(2015) displacement field differentiated by complex steps, the rate-state
right-hand side and the Cash-Karp combinations.  Rectangles are three triangles
there.
"""
import math

import numpy as np
import torch

import unicycle_b200 as ucg
from unicycle_b200 import configs

EPSILON = 1.0e-8
MAX_STEP = 1.0e4        # s; with cells of 1-2 km the error control would allow 1e5 s
FORMS = {"fp64": ucg.UCG_PREC_FP64, "split_pair": ucg.UCG_PREC_SPLIT_PAIR, "split_bf16": ucg.UCG_PREC_SPLIT_BF16,
         "hmatrix": ucg.UCG_PREC_HMATRIX, "hmatrix_split": ucg.UCG_PREC_HMATRIX_SPLIT}
HIER_LEAF = 40          # leaf size of hierarchical ensembles (at most 42)
EXACT_PATCHES = 8000    # the 64-bit restatement assembles K pair by pair


def listed():
    return [
        # a driver that keeps the state on the host and asks for one main-loop
        # iteration at a time: the reference's own loop, 512-patch fault
        dict(name="step-rect-512", path="step", mesh="rect", nx=32, nz=16),
        # the 512-rectangle strike-slip benchmark marched on the device: many
        # short steps, where launches and latency count
        dict(name="run-rect-512", path="run", mesh="rect", nx=32, nz=16, form="fp64", steps=64),
        # fault over a viscoelastic wedge, an ordinary dense model
        dict(name="run-coupled-1k-1k", path="run", mesh="coupled", nx=32, nz=32, vx=16, vy=8, vz=8, form="fp64",
             steps=16),
        # the headline megathrust, 20,000 triangles, FP64 K of 19.2 GB
        dict(name="run-tri-20000", path="run", mesh="tri", nx=100, nz=100, form="fp64", steps=4),
        # the accurate split storage on a mid-size megathrust
        dict(name="run-tri-7200-split", path="run", mesh="tri", nx=60, nz=60, form="split_pair", steps=8),
        # Green's functions of the three source families
        dict(name="assemble-rect-2048", path="assemble", mesh="rect", nx=64, nz=32, okada="fp64"),
        dict(name="assemble-tri-5000", path="assemble", mesh="tri", nx=50, nz=50, okada="fp64"),
        dict(name="assemble-coupled-1k-1k", path="assemble", mesh="coupled", nx=32, nz=32, vx=16, vy=8, vz=8,
             okada="fp64"),
        # models beyond a dense K: compression and stepping on the result
        dict(name="hbuild-tri-7200", path="hbuild", mesh="tri", nx=60, nz=60, leaf=32),
        dict(name="run-tri-7200-hmatrix", path="run", mesh="tri", nx=60, nz=60, form="hmatrix", steps=16),
        # parameter studies: 64 friction sets on one fault, dense and hierarchical
        dict(name="ens-rect-2048x64", path="ensemble", mesh="rect", nx=64, nz=32, hier=False, instances=64, steps=8),
        dict(name="ens-tri-7200x64-hier", path="ensemble", mesh="tri", nx=60, nz=60, hier=True, instances=64,
             steps=8),
    ]


def _grid(rng, lo, hi, per=1):
    """nx, nz of about a log-uniform number of patches in [lo, hi] (per patches a cell)."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi))) / per
    a = math.exp(rng.uniform(math.log(0.5), math.log(2.5)))
    nx = max(4, int(round(math.sqrt(n * a))))
    return dict(nx=nx, nz=max(4, min(int(n / nx), int(hi / per / nx))))


def draw(rng):
    k = rng.choice(["step", "run-rect", "run-tri", "run-coupled", "run-split", "asm-rect", "asm-tri", "asm-coupled",
                    "hbuild", "run-h", "ens", "ens", "ens-h"])
    if k == "step":
        m = rng.choice(["rect", "tri"])
        return dict(path="step", mesh=m, **_grid(rng, 100, 4000, 2 if m == "tri" else 1))
    if k == "run-rect":
        return dict(path="run", mesh="rect", **_grid(rng, 100, 4000), form="fp64", steps=rng.randint(8, 64))
    if k == "run-tri":
        return dict(path="run", mesh="tri", **_grid(rng, 200, 12000, 2), form="fp64", steps=rng.randint(4, 16))
    if k == "run-split":
        return dict(path="run", mesh="tri", **_grid(rng, 600, 8000, 2),
                    form=rng.choice(["split_pair", "split_bf16"]), steps=rng.randint(4, 24))
    if k in ("run-coupled", "asm-coupled"):
        c = dict(mesh="coupled", **_grid(rng, 100, 1200), vx=rng.randint(3, 16), vy=rng.randint(3, 8),
                 vz=rng.randint(3, 8))
        if k == "asm-coupled":
            return dict(path="assemble", **c, okada="fp64")
        return dict(path="run", **c, form="fp64", steps=rng.randint(8, 32))
    if k == "asm-rect":
        return dict(path="assemble", mesh="rect", **_grid(rng, 100, 5000), okada=rng.choice(["fp64", "fp64", "ref32"]))
    if k == "asm-tri":
        return dict(path="assemble", mesh="tri", **_grid(rng, 100, 8000, 2), okada="fp64")
    if k == "hbuild":
        m = rng.choice(["rect", "tri"])
        return dict(path="hbuild", mesh=m, **_grid(rng, 1000, 7200, 2 if m == "tri" else 1),
                    leaf=rng.choice([24, 32, 40]))
    if k == "run-h":
        return dict(path="run", mesh="tri", **_grid(rng, 1500, 8000, 2),
                    form=rng.choice(["hmatrix", "hmatrix_split"]), steps=rng.randint(8, 32))
    if k == "ens":
        return dict(path="ensemble", mesh="rect", **_grid(rng, 500, 4000), hier=False,
                    instances=rng.choice([8, 16, 32, 33, 48, 64, 96]), steps=rng.randint(4, 12))
    return dict(path="ensemble", mesh="tri", **_grid(rng, 1500, 7200, 2), hier=True,
                instances=rng.choice([16, 32, 50, 64]), steps=rng.randint(4, 12))


# ---- models -----------------------------------------------------------------------


def _model(case, seed):
    """Mesh, friction and initial state of a case; every random draw is the seed's."""
    if case["mesh"] == "rect":
        cfg = configs.tilt(configs.cfg1(nx=case["nx"], nz=case["nz"]))
    elif case["mesh"] == "tri":
        cfg = configs.cfg2(nx=case["nx"], nz=case["nz"], seed=seed)
    else:
        cfg = configs.cfg3(nxf=case["nx"], nzf=case["nz"], nxv=case["vx"], nyv=case["vy"], nzv=case["vz"], seed=seed)
        fr = cfg["friction"]
        fr["rake"] = np.full(cfg["n_patch"], math.radians(20.0))   # oblique: no traction that is zero by symmetry
    rng = np.random.default_rng(seed)
    cfg["y0"] = _state(cfg, cfg["friction"], rng)
    return cfg


def _state(cfg, fr, rng):
    """A state in the middle of a loading phase: slip rates around the plate rate,
    state variables near their steady state, some years of slip and the change of
    normal traction that came with it."""
    n = cfg["n_patch"]
    y = configs.steady_state(0.9 * fr["Vpl"] * np.exp(0.3 * rng.standard_normal(n)), fr)
    y[5::7] += 0.1 * rng.standard_normal(n)
    slip = 3.0 * configs.YEAR * fr["Vpl"] * np.exp(0.3 * rng.standard_normal(n))
    y[0::7], y[1::7] = slip * np.cos(fr["rake"]), slip * np.sin(fr["rake"])
    y[4::7] = 0.5 * rng.standard_normal(n)   # MPa
    if cfg.get("n_vol"):
        y = np.concatenate([y, np.zeros(12 * cfg["n_vol"])])
        for q in range(6):
            y[7 * n + q::12] = 1.0e-6 * rng.standard_normal(cfg["n_vol"])
            y[7 * n + 6 + q::12] = 0.5 * rng.standard_normal(cfg["n_vol"])   # MPa
    return y


def _friction(fr):
    return [fr[k] for k in ("Vpl", "rake", "mu0", "sig", "a", "b", "L", "Vo", "damping")]


def _geometry(cfg, coupled):
    sim = ucg.Simulation(cfg["mu"], cfg["lam"], driver="viscouscycles" if coupled else "ratestate")
    m = cfg["mesh"]
    if "rect" in m:
        sim.set_rectangles(*m["rect"])
    if "tri" in m:
        sim.set_triangles(*m["tri"])
    if coupled:
        sim.set_volumes(*m["vol"])
    sim.set_friction(*_friction(cfg["friction"]))
    if coupled:
        rh = cfg["rheology"]
        sim.set_rheology(rh["ebg"], rh["gammadot0m"], rh["npowerm"], nonlinear_maxwell=True)
    sim.set_tolerance(EPSILON, MAX_STEP)
    return sim


def _ensemble_sets(cfg, count, seed):
    """Friction of every instance and its initial state (instances x 7 patches)."""
    sets, _ = configs.parameter_sets(cfg, count, seed=1000 + seed)
    rng = np.random.default_rng(seed)
    return sets, np.stack([_state(cfg, fr, rng) for fr in sets])


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    cfg = _model(case, seed)
    s.sim = sim = _geometry(cfg, case["mesh"] == "coupled")
    s.y0 = cfg["y0"]
    form = case.get("form", "fp64")
    if case["path"] in ("step", "run"):
        if form.startswith("hmatrix"):
            sim.build_hmatrix()
        else:
            sim.buildG()
        if form != "fp64":
            sim.set_precision(FORMS[form])
            if not form.startswith("hmatrix"):
                sim.keep_fp64(False)
    elif case["path"] == "ensemble":
        if case["hier"]:
            sim.build_hmatrix(leaf=HIER_LEAF)
            sim.set_precision(ucg.UCG_PREC_HMATRIX)
        else:
            sim.buildG()
        s.ens = ens = ucg.Ensemble()
        s.geom = ens.add_geometry(sim, case["instances"])
        sim.close()
        sets, s.y0 = _ensemble_sets(cfg, case["instances"], seed)
        for i, fr in enumerate(sets):
            ens.set_friction(s.geom, i, *_friction(fr))
        ens.set_tolerance(EPSILON, MAX_STEP)
    return s


def run(s):
    c, sim = s.case, s.sim
    if c["path"] == "assemble":
        sim.buildG(ucg.UCG_OKADA_REF32IO if c["okada"] == "ref32" else ucg.UCG_OKADA_FP64)
        dydt, vmax = sim.odefun(s.y0)
        return {"dydt": dydt, "vmax": vmax}
    if c["path"] == "hbuild":
        sim.build_hmatrix(leaf=c["leaf"])
        sim.set_precision(ucg.UCG_PREC_HMATRIX)
        dydt, vmax = sim.odefun(s.y0)
        return {"dydt": dydt, "vmax": vmax}
    if c["path"] == "step":
        t, y, dydt, dt_next, dt_done, rejected = sim.step(0.0, s.y0, MAX_STEP)
        return {"y": y, "dydt": dydt, "time": t, "dt_next": dt_next, "rejected": rejected}
    if c["path"] == "run":
        sim.set_state(s.y0, 0.0, MAX_STEP)
        steps = sim.run(1.0e30, c["steps"])
        y, t, dt_next, _, _ = sim.get_state()
        return {"y": y, "time": t, "dt_next": dt_next, "steps": steps}
    s.ens.set_states(s.geom, s.y0, 0.0, MAX_STEP)
    s.ens.run(1.0e30, c["steps"])
    y, t, dt_next, accepted, rejected, status = s.ens.get_states(s.geom)
    return {"y": y, "time": t, "dt_next": dt_next, "accepted": accepted, "rejected": rejected, "status": status}


# ---- work -------------------------------------------------------------------------


def _sizes(case):
    np_ = case["nx"] * case["nz"] * (2 if case["mesh"] == "tri" else 1)
    nv = case["vx"] * case["vy"] * case["vz"] if case["mesh"] == "coupled" else 0
    return np_, nv, 2 * np_ + 6 * nv, 3 * np_ + 6 * nv


# operations of one (receiver, source) pair when every closed form is evaluated
# once, with its gradient and all the source's unit components together
PAIR_FLOPS = {"rect": 4.0e3, "tri": 7.0e3, "vol": 4.0e4}


def _hier_bytes(n_patch):
    """FP64 bytes of the hierarchical K, which grow as N^1.58 over 7,200-80,000 triangles."""
    return min(2.99e9 * (n_patch / 20000.0) ** 1.58, 48.0 * n_patch * n_patch)


def work(case):
    np_, nv, n, m = _sizes(case)
    state = 8.0 * (7 * np_ + 12 * nv)
    if case["path"] in ("assemble", "hbuild"):
        e = np_ + nv
        flops = e * (np_ * PAIR_FLOPS["tri" if case["mesh"] == "tri" else "rect"] + nv * PAIR_FLOPS["vol"])
        stored = _hier_bytes(np_) if case["path"] == "hbuild" else 8.0 * m * n
        return {"bytes": 2 * stored + 2 * state, "flops": flops + 2.0 * m * n}
    if case["path"] == "ensemble":
        k = _hier_bytes(np_) / 2 if case["hier"] else 4.0 * m * n
        i = case["instances"]
        return {"bytes": case["steps"] * 6 * (k + 4.0 * i * (n + m) + 2 * i * state),
                "flops": case["steps"] * 6 * i * (k / 2)}
    steps = case.get("steps", 1)
    form = case.get("form", "fp64")
    if form.startswith("hmatrix"):
        k = _hier_bytes(np_) / (2 if form == "hmatrix_split" else 1)
        one = 6 * k
        flops = 6 * 2.0 * _hier_bytes(np_) / 8
    else:
        one = {"fp64": 48.0, "split_pair": 24.0, "split_bf16": 14.0}[form] * m * n
        flops = 12.0 * m * n
    return {"bytes": steps * (one + 6 * 2 * state), "flops": steps * flops}


# ---- the same in 64 bits, with torch alone ----------------------------------------

_STEP = 1.0e-30   # imaginary step: derivatives to rounding


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _arctan2(n, d):
    """1j times the differential of atan2(n, d): only gradients are formed, no value."""
    return 1j * (d.real * n.imag - n.real * d.imag) / (n.real ** 2 + d.real ** 2)


def _log(a):
    return 1j * a.imag / a.real


def _angular(x, y, z, tv, side, cos_a, sin_a, by, bz, nu):
    """Displacement of one angular dislocation in the frame of its triangle, (by, bz) pairs."""
    a00, a01, a10, a11 = side[1], -side[0], side[0], side[1]
    ty, tz = y - tv[0], z - tv[1]
    y1, z1 = a00 * ty + a01 * tz, a10 * ty + a11 * tz
    zeta = y1 * sin_a + z1 * cos_a
    r = torch.sqrt(x * x + y1 * y1 + z1 * z1)
    p, q = 1.0 / (r * (r - zeta)), 1.0 / (r * (r - z1))
    lz, le = _log(r - z1), _log(r - zeta)
    k, m = 1.0 / (8.0 * math.pi * (1.0 - nu)), 1.0 - 2.0 * nu
    uy = k * (x * x * (cos_a * p - q) - m * (cos_a * le - lz))
    vy = k * x * (y1 * cos_a * p - sin_a * cos_a * r * p - y1 * q)
    wy = k * x * (z1 * cos_a * p - cos_a * cos_a * r * p + 1.0 / r)
    uz = k * sin_a * (m * le - x * x * p)
    vz = k * sin_a * x * (sin_a * r * p - y1 * p)
    wz = k * sin_a * x * (cos_a * r * p - z1 * p)
    out = []
    for b_y, b_z in zip(by, bz):
        c, d = a00 * b_y + a01 * b_z, a10 * b_y + a11 * b_z
        v, w = c * vy + d * vz, c * wy + d * wz
        out.append((c * uy + d * uz, a00 * v + a10 * w, a01 * v + a11 * w))
    return out


def _unit(v):
    return v / torch.sqrt((v * v).sum(-1, keepdim=True))


def _triangle(X, P, b, nu):
    """Full-space displacement (east, north, up) of triangles P at X for slips b (modes, n, 3)."""
    p1, p2, p3 = P
    vn = _unit(torch.linalg.cross(p2 - p1, p3 - p1))
    vs = torch.stack([-vn[:, 1], vn[:, 0], torch.zeros_like(vn[:, 0])], -1)
    vs = _unit(vs)
    vd = torch.linalg.cross(vn, vs)

    def local(w):
        return [sum(w[c] * f[:, c] for c in range(3)) for f in (vn, vs, vd)]

    x, y, z = local([X[c] - p2[:, c] for c in range(3)])
    q1, q3 = ([(f * (p - p2)).sum(-1) for f in (vs, vd)] for p in (p1, p3))

    def side(u, v):
        d = torch.stack([v[0] - u[0], v[1] - u[1]])
        return d / torch.sqrt((d * d).sum(0))

    q2 = [torch.zeros_like(q1[0])] * 2
    e12, e13, e23 = side(q1, q2), side(q1, q3), side(q2, q3)
    A = torch.acos((e12 * e13).sum(0)) - math.pi
    B = torch.acos(-(e12 * e23).sum(0)) - math.pi
    C = torch.acos((e23 * e13).sum(0)) - math.pi
    # which configuration of the legs leaves no artefact here: barycentric regions
    yy, zz = y.real, z.real
    den = -q3[1] * (q1[0] - q3[0]) + q3[0] * (q1[1] - q3[1])
    a = (-q3[1] * (yy - q3[0]) + q3[0] * (zz - q3[1])) / den
    bb = ((q3[1] - q1[1]) * (yy - q3[0]) + (q1[0] - q3[0]) * (zz - q3[1])) / den
    c = 1.0 - a - bb
    neg = ((a <= 0) & (bb > c) & (c > a)) | ((bb <= 0) & (c > a) & (a > bb)) | ((c <= 0) & (a > bb) & (bb > c))
    sg = torch.where(neg, -1.0, 1.0).to(torch.float64)
    by, bz = [(m * vs).sum(-1) for m in b], [(m * vd).sum(-1) for m in b]
    total = [[0.0, 0.0, 0.0] for _ in b]
    for tv, e, s, ang in ((q1, e13, -sg, A), (q2, e12, sg, B), (q3, e23, sg, C)):
        for t, w in zip(total, _angular(x, y, z, tv, s * e[:, None], torch.cos(ang), torch.sin(ang), by,
                                        bz, nu)):
            for k in range(3):
                t[k] = t[k] + w[k]
    r1, r2, r3 = [-x, q1[0] - y, q1[1] - z], [-x, -y, -z], [-x, q3[0] - y, q3[1] - z]

    def dot(u, v):
        return u[0] * v[0] + u[1] * v[1] + u[2] * v[2]

    n1, n2, n3 = (torch.sqrt(dot(r, r)) for r in (r1, r2, r3))
    num = (r1[0] * (r2[1] * r3[2] - r2[2] * r3[1]) - r1[1] * (r2[0] * r3[2] - r2[2] * r3[0])
           + r1[2] * (r2[0] * r3[1] - r2[1] * r3[0]))
    solid = _arctan2(num, n1 * n2 * n3 + dot(r1, r2) * n3 + dot(r1, r3) * n2 + dot(r2, r3) * n1) / (-2.0 * math.pi)
    out = []
    for t, b_y, b_z in zip(total, by, bz):
        t = [t[0], t[1] + solid * b_y, t[2] + solid * b_z]
        out.append([t[0] * vn[:, k] + t[1] * vs[:, k] + t[2] * vd[:, k] for k in range(3)])
    return out


def _free_surface(y1, y2, y3, sb, cb, a, b, nu):
    """Harmonic displacement of one angular dislocation with a vertical leg; b = (b1, b2, b3)."""
    y3b = y3 + 2.0 * a
    z1b, z3b = y1 * cb + y3b * sb, -y1 * sb + y3b * cb
    r = torch.sqrt(y1 * y1 + y2 * y2 + y3b * y3b)
    ct, m, n = cb / sb, 1.0 - 2.0 * nu, 1.0 - nu
    fi = 2.0 * _arctan2(-y2, -(r + y3b) * ((1.0 + cb) / sb) + y1)
    ry, rz, ya = r + y3b, r + z3b, y3 + a
    w, s = r * cb + y3b, r * sb - y1
    ly, lz = _log(ry), _log(rz)
    ca, ar = cb + a / r, a / r
    sc = 1.0 + a / (r * cb)
    v11 = (-2 * n * m * fi * ct ** 2 + m * y2 / ry * ((m - ar) * ct - y1 / ry * (nu + ar))
           + m * y2 * cb * ct / rz * ca + a * y2 * ya * ct / r ** 3
           + y2 * ya / (r * ry) * (-m * ct + y1 / ry * (2 * nu + ar) + a * y1 / r ** 2)
           + y2 * ya / (r * rz) * (cb / rz * (w * (m * cb - ar) * ct + 2 * n * s * cb) - a * y3b * cb * ct / r ** 2))
    v21 = (m * ((2 * n * ct ** 2 - nu) * ly - (2 * n * ct ** 2 + m) * cb * lz)
           - m / ry * (y1 * ct * (m - ar) + nu * y3b - a + y2 ** 2 / ry * (nu + ar))
           - m * z1b * ct / rz * ca - a * y1 * ya * ct / r ** 3
           + ya / ry * (-2 * nu + 1 / r * (m * y1 * ct - a) + y2 ** 2 / (r * ry) * (2 * nu + ar) + a * y2 ** 2 / r ** 3)
           + ya / rz * (cb ** 2 - 1 / r * (m * z1b * ct + a * cb) + a * y3b * z1b * ct / r ** 3
                        - 1 / (r * rz) * (y2 ** 2 * cb ** 2 - a * z1b * ct / r * w)))
    v31 = (2 * n * (m * fi * ct + y2 / ry * (2 * nu + ar) - y2 * cb / rz * ca)
           + y2 * ya / r * (2 * nu / ry + a / r ** 2)
           + y2 * ya * cb / (r * rz) * (1 - 2 * nu - w / rz * ca - a * y3b / r ** 2))
    v12 = (m * ((2 * n * ct ** 2 + nu) * ly - (2 * n * ct ** 2 + 1) * cb * lz)
           + m / ry * (-m * y1 * ct + nu * y3b - a + a * y1 * ct / r + y1 ** 2 / ry * (nu + ar))
           - m * ct / rz * (z1b * cb - a * s / (r * cb)) - a * y1 * ya * ct / r ** 3
           + ya / ry * (2 * nu + 1 / r * (m * y1 * ct + a) - y1 ** 2 / (r * ry) * (2 * nu + ar) - a * y1 ** 2 / r ** 3)
           + ya * ct / rz * (-cb * sb + a * y1 * y3b / (r ** 3 * cb) + s / r * (2 * n * cb - w / rz * sc)))
    v22 = (2 * n * m * fi * ct ** 2 + m * y2 / ry * (-(m - ar) * ct + y1 / ry * (nu + ar))
           - m * y2 * ct / rz * sc - a * y2 * ya * ct / r ** 3
           + y2 * ya / (r * ry) * (m * ct - 2 * nu * y1 / ry - a * y1 / r * (1 / r + 1 / ry))
           + y2 * ya * ct / (r * rz) * (-2 * n * cb + w / rz * sc + a * y3b / (r ** 2 * cb)))
    v32 = (-2 * n * m * ct * (ly - cb * lz) - 2 * n * y1 / ry * (2 * nu + ar) + 2 * n * z1b / rz * ca
           + ya / r * (m * ct - 2 * nu * y1 / ry - a * y1 / r ** 2)
           - ya / rz * (cb * sb + w * ct / r * (2 * n * cb - w / rz)
                        + ar * (sb - y3b * z1b / r ** 2 - z1b * w / (r * rz))))
    v13 = (m * (y2 / ry * (1 + ar) - y2 * cb / rz * ca) - y2 * ya / r * (a / r ** 2 + 1 / ry)
           + y2 * ya * cb / (r * rz) * (w / rz * ca + a * y3b / r ** 2))
    v23 = (m * (-sb * lz - y1 / ry * (1 + ar) + z1b / rz * ca) + y1 * ya / r * (a / r ** 2 + 1 / ry)
           - ya / rz * (sb * (cb - ar) + z1b / r * (1 + a * y3b / r ** 2)
                        - 1 / (r * rz) * (y2 ** 2 * cb * sb - a * z1b / r * w)))
    v33 = (2 * n * fi + 2 * n * y2 * sb / rz * ca
           + y2 * ya * sb / (r * rz) * (1 + w / rz * ca + a * y3b / r ** 2))
    k = 1.0 / (4.0 * math.pi * n)
    return [[k * (g[0] * v11 + g[1] * v12 + g[2] * v13), k * (g[0] * v21 + g[1] * v22 + g[2] * v23),
             k * (g[0] * v31 + g[1] * v32 + g[2] * v33)] for g in b]


def _harmonic(X, PA, PB, b, nu):
    """Free-surface term of one triangle side, (east, north, up)."""
    sv = PB - PA
    beta = torch.acos(-sv[:, 2] / torch.sqrt((sv * sv).sum(-1)))
    e1 = _unit(sv[:, :2])
    e2 = torch.stack([e1[:, 1], -e1[:, 0]], -1)

    def local(w):
        return [e1[:, 0] * w[0] + e1[:, 1] * w[1], e2[:, 0] * w[0] + e2[:, 1] * w[1], -w[2]]

    ya = local([X[c] - PA[:, c] for c in range(3)])
    yb = local([X[c] - PB[:, c] for c in range(3)])
    s = torch.where(ya[0].real >= 0, -1.0, 1.0).to(torch.float64)   # mirrored frame, angle pi - beta
    sb, cb = torch.sin(beta), torch.cos(beta) * s
    bl = [local([m[:, c] for c in range(3)]) for m in b]
    bl = [(g[0] * s, g[1] * s, g[2]) for g in bl]
    out = []
    for va, vb in zip(_free_surface(s * ya[0], s * ya[1], ya[2], sb, cb, -PA[:, 2], bl, nu),
                      _free_surface(s * yb[0], s * yb[1], yb[2], sb, cb, -PB[:, 2], bl, nu)):
        v = [s * (vb[0] - va[0]), s * (vb[1] - va[1]), vb[2] - va[2]]
        out.append([e1[:, 0] * v[0] + e2[:, 0] * v[1], e1[:, 1] * v[0] + e2[:, 1] * v[1], -v[2]])
    return out


def _half_space(X, P, b, nu):
    mirror = torch.tensor([1.0, 1.0, -1.0], dtype=torch.float64, device=P[0].device)
    # the image keeps the real triangle's slip in its own (mirrored) frame
    parts = [_triangle(X, P, b, nu), _triangle(X, [p * mirror for p in P], [_mirrored(m, P, mirror) for m in b], nu)]
    for k in range(3):
        parts.append(_harmonic(X, P[k], P[(k + 1) % 3], b, nu))
    return [[sum(p[m][c] for p in parts) for c in range(3)] for m in range(len(b))]


def _frame(P):
    vn = _unit(torch.linalg.cross(P[1] - P[0], P[2] - P[0]))
    vs = _unit(torch.stack([-vn[:, 1], vn[:, 0], torch.zeros_like(vn[:, 0])], -1))
    return vs, torch.linalg.cross(vn, vs)


def _mirrored(b, P, mirror):
    (s, d), (s2, d2) = _frame(P), _frame([p * mirror for p in P])
    return (b * s).sum(-1, keepdim=True) * s2 + (b * d).sum(-1, keepdim=True) * d2


def _patches(cfg):
    """Receiver centres and frames (NED), and the source triangles with their slip vectors."""
    if "rect" in cfg["mesh"]:
        x, L, W, st, dp = cfg["mesh"]["rect"]
        s = np.stack([np.cos(st), np.sin(st), 0 * st], 1)
        d = np.stack([np.sin(st) * np.cos(dp), -np.cos(st) * np.cos(dp), -np.sin(dp)], 1)
        n = np.stack([-np.sin(st) * np.sin(dp), np.cos(st) * np.sin(dp), -np.cos(dp)], 1)
        a, w = L[:, None] * s, -W[:, None] * d
        # three triangles with the centre inside one of them
        p0, e, p1, p2, p3 = x, x + 0.5 * a, x + a, x + a + w, x + w
        return x + 0.5 * a + 0.5 * w, s, d, n, [(p0, e, p3), (e, p1, p2), (e, p2, p3)]
    i1, i2, i3, v = cfg["mesh"]["tri"]
    A, B, C = v[i1 - 1], v[i2 - 1], v[i3 - 1]
    n = np.cross(B - A, C - A)
    n /= np.linalg.norm(n, axis=1)[:, None]
    n = np.where(n[:, 2:] > 0, -n, n)
    s = np.stack([n[:, 1], -n[:, 0]], 1) / np.linalg.norm(n[:, :2], axis=1)[:, None]
    s = np.concatenate([s, np.zeros((len(s), 1))], 1)
    return (A + B + C) / 3.0, s, np.cross(n, s), n, [(A, B, C)]


def _exact_k(cfg):
    """K (3 receivers x 2 sources, rows ts, td, tn) by complex-step differentiation."""
    dev, f64 = _device(), torch.float64
    mu, lam = cfg["mu"], cfg["lam"]
    nu = lam / (lam + mu) / 2.0
    xc, s, d, n, tris = _patches(cfg)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=f64, device=dev)  # noqa: E731
    enu = lambda a: t(np.stack([a[:, 1], a[:, 0], -a[:, 2]], 1))  # noqa: E731
    R = [t(a) for a in (s, d, n)]
    # the field's jump follows each triangle's own normal: slip of the hanging
    # wall along s and d, signed by that normal against n
    sources = []
    for P in tris:
        pe = [enu(p) for p in P]
        vn = torch.linalg.cross(pe[1] - pe[0], pe[2] - pe[0])
        sign = torch.sign((vn * enu(n)).sum(-1, keepdim=True))
        sources.append((pe, [sign * enu(s), sign * enu(d)]))
    N = len(xc)
    X = enu(xc)
    K = torch.empty((3 * N, 2 * N), dtype=f64, device=dev)
    rows = max(1, 2_000_000 // N)
    for r0 in range(0, N, rows):
        r1 = min(N, r0 + rows)
        g = [[[None] * 3 for _ in range(3)] for _ in range(2)]
        for j in range(3):
            Z = [X[r0:r1, c:c + 1] + (1j * _STEP if c == j else 0j) for c in range(3)]
            u = [[0.0] * 3 for _ in range(2)]
            for pe, b in sources:
                for m, w in enumerate(_half_space(Z, pe, b, nu)):
                    for c in range(3):
                        u[m][c] = u[m][c] + w[c].imag / _STEP
            for m in range(2):
                for c in range(3):
                    g[m][c][j] = u[m][c]
        to = (1, 0, 2)            # ENU -> NED, the vertical changes sign
        sg = (1.0, 1.0, -1.0)
        for m in range(2):
            e = [[0.5 * sg[a] * sg[b] * (g[m][to[a]][to[b]] + g[m][to[b]][to[a]]) for b in range(3)] for a in range(3)]
            tr = lam * (e[0][0] + e[1][1] + e[2][2])
            nn = R[2][r0:r1]
            T = [sum((2.0 * mu * e[a][b] + (tr if a == b else 0.0)) * nn[:, b:b + 1] for b in range(3))
                 for a in range(3)]
            for q in range(3):
                f = R[q][r0:r1]
                K[3 * r0 + q:3 * r1:3, m::2] = sum(T[a] * f[:, a:a + 1] for a in range(3))
    return K


def _rhs(K, fr, y):
    """dydt of states y (instances, patches, 7); friction arrays (instances, patches)."""
    lg = math.log(10.0)
    rake, V = torch.atan2(y[..., 3], y[..., 2]), torch.exp(y[..., 6] * lg)
    cr, sr = torch.cos(rake), torch.sin(rake)
    v = torch.stack([V * cr - fr["Vpl"] * torch.cos(fr["rake"]), V * sr - fr["Vpl"] * torch.sin(fr["rake"])], -1)
    t = (K @ v.reshape(len(y), -1).T).T.reshape(len(y), -1, 3)
    dth = (torch.exp(-y[..., 5] * lg) - V / fr["L"]) / lg
    dv = (t[..., 0] * cr + t[..., 1] * sr - fr["b"] * fr["sig"] * dth * lg) / (fr["a"] * fr["sig"]
                                                                             + fr["damping"] * V) / lg
    corr = fr["damping"] * V * dv * lg
    return torch.stack([V * cr, V * sr, t[..., 0] - corr * cr, t[..., 1] - corr * sr, t[..., 2], dth, dv], -1)


_CK = [[], [0.2], [3 / 40, 9 / 40], [0.3, -0.9, 1.2], [-11 / 54, 2.5, -70 / 27, 35 / 27],
       [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]]
_CKC = [37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771]


def exact(case, seed):
    np_, _, _, _ = _sizes(case)
    if case["mesh"] == "coupled" or np_ > EXACT_PATCHES:
        return None   # no short closed form of the cuboids; K of the largest model takes too long
    cfg = _model(case, seed)
    if case["path"] == "ensemble":
        sets, y0 = _ensemble_sets(cfg, case["instances"], seed)
    else:
        sets, y0 = [cfg["friction"]], cfg["y0"][None]
    dev = _device()
    fr = {k: torch.as_tensor(np.stack([f[k] for f in sets]), device=dev) for k in sets[0]}
    K = _exact_k(cfg)
    y = torch.as_tensor(y0, device=dev).reshape(len(sets), np_, 7)
    k1 = _rhs(K, fr, y)
    flat = (lambda a: a.reshape(len(sets), -1).cpu().numpy()) if case["path"] == "ensemble" else (
        lambda a: a.reshape(-1).cpu().numpy())
    if case["path"] in ("assemble", "hbuild"):
        return {"dydt": flat(k1), "vmax": float(torch.exp(y[..., 6] * math.log(10.0)).max())}
    h, steps = MAX_STEP, case.get("steps", 1)
    for _ in range(steps):
        k = [_rhs(K, fr, y)]
        for c in _CK[1:]:
            k.append(_rhs(K, fr, y + h * sum(a * b for a, b in zip(c, k))))
        y = y + h * sum(a * b for a, b in zip(_CKC, k))
    t = h * steps
    if case["path"] == "step":
        return {"y": flat(y), "dydt": flat(k1), "time": t, "dt_next": h, "rejected": None}
    if case["path"] == "run":
        return {"y": flat(y), "time": t, "dt_next": h, "steps": None}
    one = np.ones(len(sets))
    return {"y": flat(y), "time": t * one, "dt_next": h * one, "accepted": None, "rejected": None, "status": None}
