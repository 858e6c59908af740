"""ewpt_gauss_project where its index arithmetic and its small solve can go
wrong: the smallest and odd lattices (fewer staggered modes, rows shorter and
longer than a warp), and a uniform Higgs field, whose generator overlaps make
the solve rank-deficient.  Against ewpt/ic.py gauss_project to 1e-9 of each
array's largest value, the bar of the other comparison with it."""
import numpy as np
import pytest

import ewpt
from ewpt import ic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build_lib

    build_lib.build()


@pytest.mark.parametrize("uniform", [False, True])
@pytest.mark.parametrize("shape", [(7, 7, 7), (9, 8, 7), (8, 8, 8), (34, 9, 13), (65, 8, 10)])
def test_matches_the_host_projection(shape, uniform):
    p = ewpt.baseline_couplings(shape=shape, N=shape[0], dx=0.25, dt=0.025)
    y0 = ic.thermal(shape, p.dx, T=1.5, gw=p.gw, gy=p.gy, seed=sum(shape), gauss_iters=0, with_momenta=True)
    if uniform:
        y0[0:4] = np.array([0.6, 0.0, 0.8, 0.0])[:, None]
    yh = ic.gauss_project(y0.copy(), shape, p.dx, p.gw, p.gy, iters=3)
    with ewpt.Lattice(p) as lat:
        lat.set_state(y0)
        lat.gauss_project(3)
        yd = lat.get_state()
    np.testing.assert_array_equal(yd[:20], y0[:20])
    scale = np.abs(yh[20:]).max(axis=1, keepdims=True)
    assert (np.abs(yd[20:] - yh[20:]) / scale).max() < 1e-9
