"""Triangle assembly per mesh edge: the free-surface term is formed once per edge
and shared by the edge's triangles, in batches of receivers.

Checked against the oracle where that can go wrong: one triangle pair, meshes that
end inside a CTA, more receivers than one batch holds (1,200 triangles), vertices
that are not shared, windings that run along a shared edge the same way, vertical
edges (whose term vanishes) and volume receivers (6 rows).

Tolerance: |K - K_ref| <= 1e-12 of the largest entry in the receiver's rows, the
bound of the FP64 assembly (both sides round at about 3e-13 there)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _split(v, i1, i2, i3):
    """The same triangles on vertices of their own."""
    n = len(i1)
    w = np.stack([v[i1 - 1], v[i2 - 1], v[i3 - 1]], 1).reshape(-1, 3)
    k = 3 * np.arange(n)
    return w, k + 1, k + 2, k + 3


def _flip(i1, i2, i3):
    """Every second triangle wound the other way."""
    i2, i3 = i2.copy(), i3.copy()
    i2[::2], i3[::2] = i3[::2].copy(), i2[::2].copy()
    return i1, i2, i3


def _vertical(nx, nz, h=900.0):
    g = lambda i, k: i * (nz + 1) + k + 1  # noqa: E731
    v = np.array([[i * h, 30.0, 500.0 + k * h] for i in range(nx + 1) for k in range(nz + 1)])
    t = [(g(i, k), g(i + 1, k), g(i + 1, k + 1)) for i in range(nx) for k in range(nz)]
    t += [(g(i, k), g(i + 1, k + 1), g(i, k + 1)) for i in range(nx) for k in range(nz)]
    i1, i2, i3 = (np.array(c) for c in zip(*t))
    return v, i1, i2, i3


def _mesh(kind, nx, nz):
    from unicycle_b200 import configs
    if kind == "vertical":
        return _vertical(nx, nz)
    i1, i2, i3, v = configs.megathrust_mesh(nx, nz)
    if kind == "split":
        return _split(v, i1, i2, i3)
    if kind == "flip":
        return (v,) + _flip(i1, i2, i3)
    return v, i1, i2, i3


@pytest.mark.parametrize("kind,nx,nz", [("shared", 1, 1), ("shared", 5, 13), ("shared", 30, 20), ("split", 4, 3),
                                        ("flip", 9, 7), ("vertical", 4, 3)])
def test_tri_assembly(ucg, oracle_lib, kind, nx, nz):
    v, i1, i2, i3 = _mesh(kind, nx, nz)
    sim = ucg.Simulation(3.0e4, 2.4e4)
    sim.set_triangles(i1, i2, i3, v)
    sim.buildG()
    K = sim.copy_G()
    sim.close()
    ref = oracle_lib.Mesh(3.0e4, 2.4e4, tri=(v, i1, i2, i3)).build_g()
    scale = np.repeat(np.abs(ref).reshape(-1, 3, ref.shape[1]).max(axis=(1, 2)), 3)[:, None]
    assert np.max(np.abs(K - ref) / scale) < 1e-12


def test_tri_sources_volume_receivers(ucg, oracle_lib):
    v, i1, i2, i3 = _mesh("shared", 3, 4)
    x = np.array([[1000.0, 20e3, 60e3], [9000.0, 45e3, 70e3]])
    vol = (x, np.full(2, 3e3), np.full(2, 2e3), np.full(2, 2.5e3), np.radians([0.0, 35.0]))
    sim = ucg.Simulation(3.0e4, 3.0e4, driver="viscouscycles")
    sim.set_triangles(i1, i2, i3, v)
    sim.set_volumes(*vol)
    sim.buildG()
    n = 2 * len(i1)
    K = sim.copy_G()[:, :n]
    sim.close()
    ref = oracle_lib.Mesh(3.0e4, 3.0e4, tri=(v, i1, i2, i3), vol=vol).build_g()[:, :n]
    r = 3 * len(i1)
    for a, b, dof in ((K[:r], ref[:r], 3), (K[r:], ref[r:], 6)):
        scale = np.repeat(np.abs(b).reshape(-1, dof, n).max(axis=(1, 2)), dof)[:, None]
        assert np.max(np.abs(a - b) / scale) < 1e-12
