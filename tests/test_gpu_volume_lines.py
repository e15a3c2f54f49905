"""Volume columns of K at receivers next to the line through a cuboid's vertical edge,
above and below the cuboid.  The stress is smooth there, while each corner's terms
grow with the inverse (square) of the distance to the line: what grows has to cancel
before it is formed, not in the sum over the corners.

Against Mindlin's point force integrated over the cuboid's faces (oracle/mindlin.cc),
which knows no such line.  Tolerance: 4e-8 of the receiver's scale, the bound of the
two routes elsewhere (their own agreement is 1e-9)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MU, LAM = 3.0e4, 2.6e4
L, T, W, Q3 = 3100.0, 2300.0, 1700.0, 2900.0


@pytest.mark.parametrize("strike", [0.0, 0.7])
@pytest.mark.parametrize("off", [1e-6, 1e-3, 1.0])
def test_receivers_next_to_a_vertical_edge_line(ucg, oracle_lib, strike, off):
    q = np.array([1300.0, -700.0, Q3])
    vol = (q[None], np.full(1, L), np.full(1, T), np.full(1, W), np.full(1, strike))
    c, s = np.cos(strike), np.sin(strike)
    size, dip = 200.0, np.radians(50.0)
    x = []
    for k, depth in enumerate((0.35 * Q3, 0.8 * Q3, Q3 + 1.4 * W, Q3 + 2.7 * W)):
        for a in (0.0, L):
            for b in (-T / 2, T / 2):
                phi = 0.9 + 1.1 * k + a + b      # direction of the offset
                f, g = a + off * np.cos(phi), b + off * np.sin(phi)
                x.append([q[0] + f * c - g * s, q[1] + f * s + g * c, depth])
    n = len(x)
    # a patch's centre lies half its length along strike (north) and half its width down dip (east and down)
    corner = np.array(x) - [size / 2, np.cos(dip) * size / 2, np.sin(dip) * size / 2]
    rect = (corner, np.full(n, size), np.full(n, size), np.zeros(n), np.full(n, dip))
    M = oracle_lib.Mesh(MU, LAM, rect=rect, vol=vol)
    assert np.max(np.abs(M.rect_frames[3] - np.array(x))) < 1e-9
    oracle_lib.set_volume_route(1)
    try:
        G = M.build_g()[:3 * n, 2 * n:]
    finally:
        oracle_lib.set_volume_route(0)
    sim = ucg.Simulation(MU, LAM, driver="viscouscycles")
    sim.set_rectangles(*rect)
    sim.set_volumes(*vol)
    sim.buildG()
    K = sim.copy_G()[:3 * n, 2 * n:]
    sim.close()
    assert np.all(np.isfinite(G)) and np.all(np.isfinite(K))
    scale = np.abs(G).reshape(n, -1).max(axis=1)
    assert np.max(np.abs(K - G).reshape(n, -1).max(axis=1) / scale) < 4e-8
