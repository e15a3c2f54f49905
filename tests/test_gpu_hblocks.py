"""Block assembly of the hierarchical matrix: all blocks of a batch in one launch.

The product with H against the dense K of the same model, where tiles of blocks
can go wrong: a single dense block (one tile, no low-rank block), leaves that do
not divide a tile, odd patch counts, the smallest leaf size (4), both patch families and
the REAL*4 interface.

Tolerance: every low-rank block is checked to 10 eps of its own product at the
build (dense ones are exact), so |H x - K x| <= 10 eps sum |K| |x| per row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 1.0e-6


@pytest.mark.parametrize("family,nx,nz,leaf,mode", [("tri", 1, 1, 32, 0), ("tri", 7, 5, 11, 0), ("tri", 19, 13, 32, 0),
                                                    ("rect", 5, 5, 32, 0), ("rect", 23, 11, 17, 0),
                                                    ("rect", 16, 9, 24, 1), ("tri", 4, 3, 4, 0)])
def test_product_matches_dense(ucg, family, nx, nz, leaf, mode):
    from unicycle_b200 import configs
    cfg = configs.cfg2(nx=nx, nz=nz) if family == "tri" else configs.tilt(configs.cfg1(nx=nx, nz=nz))
    sim = ucg.Simulation(cfg["mu"], cfg["lam"])
    (sim.set_triangles if family == "tri" else sim.set_rectangles)(*cfg["mesh"][family])
    sim.buildG(mode)
    K = sim.copy_G()
    sim.build_hmatrix(mode, eps=EPS, leaf=leaf)
    x = np.random.default_rng(nx).standard_normal(K.shape[1])
    y = sim.hmatrix_matvec(x)
    sim.close()
    assert np.all(np.abs(y - K @ x) <= 10 * EPS * (np.abs(K) @ np.abs(x)))
