"""The 6th-order FP64 stages keep to the bit what their equations keep."""
import math

import numpy as np
import pytest

import ewpt

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build_lib

    build_lib.build()


def state(shape, seed, kind="random"):
    if kind == "bubbles":
        p = ewpt.baseline_couplings(shape=shape, N=shape[0])
        return ewpt.ic.bubbles_tanh(shape, p.dx, 3, seed=seed)
    rng = np.random.default_rng(seed)
    y = 0.1 * rng.normal(size=(36, math.prod(shape)))
    y[0] += 1.0
    y[21][rng.random(y.shape[1]) < 0.3] = 0.0
    return y


def evolve(shape, y, steps=3, **couplings):
    with ewpt.Lattice(ewpt.baseline_couplings(shape=shape, N=shape[0], **couplings)) as lat:
        lat.set_state(y)
        lat.step(steps, Jex=0.0, gamma=0.01)
        return lat.get_state()


@pytest.mark.parametrize("kind", ["random", "bubbles"])
@pytest.mark.parametrize("beta", [0.0, 0.3])
def test_minus_phi_evolves_to_minus_phi(kind, beta):
    """The equations keep Phi -> -Phi (gauge fields unchanged), and so do the
    roundings: both runs agree to the bit."""
    shape = (24, 18, 20)
    y = state(shape, 6, kind)
    higgs = [0, 1, 2, 3, 20, 21, 22, 23]
    sign = np.ones((36, 1))
    sign[higgs] = -1.0
    a = evolve(shape, y, beta_w=beta, beta_y=beta)
    b = evolve(shape, np.where(y == 0.0, 0.0, sign * y), beta_w=beta, beta_y=beta)
    assert np.isfinite(a).all()
    np.testing.assert_array_equal(b, sign * a)


def test_a_mirror_image_evolves_to_the_mirror_image():
    """x -> -x: the x components of the gauge fields and momenta change sign."""
    shape = (20, 9, 14)
    y = state(shape, 8)
    sign = np.ones((36, 1, 1, 1))
    sign[[4, 7, 10, 13, 24, 27, 30, 33]] = -1.0

    def mirror(v):
        w = sign * v.reshape(36, *shape[::-1])[..., ::-1]
        return np.where(w == 0.0, 0.0, w).reshape(36, -1)

    a = evolve(shape, y)
    np.testing.assert_array_equal(evolve(shape, mirror(y)), mirror(a))


# 32-site blocks that straddle the edges of planes, of the host step's windows
# and of slabs, where a whole lattice's blocks lie otherwise
@pytest.mark.parametrize("shape", [(7, 9, 40), (11, 13, 37), (33, 7, 33)])
@pytest.mark.parametrize("beta", [0.0, 0.3])
def test_windows_and_slabs_of_ragged_planes(shape, beta):
    import torch

    from ewpt.slabs import SlabGroup

    p = ewpt.baseline_couplings(shape=shape, N=shape[0], beta_w=beta, beta_y=-beta)
    y = state(shape, 5)
    ref = evolve(shape, y, steps=2, beta_w=beta, beta_y=-beta)
    for cut in ([3, shape[2] - 3], [5, 7, shape[2] - 12]):
        with SlabGroup(p, len(cut), nz_local=cut) as g:
            g.set_state(y)
            g.step(2, Jex=0.0, gamma=0.01)
            np.testing.assert_array_equal(g.get_state(), ref)
    with ewpt.Lattice(p) as lat:
        lat.set_state(y)
        lat.step(2)
        ref = lat.get_state()
    with ewpt.Lattice(p) as lat:
        src = torch.from_numpy(y).pin_memory()
        dst = torch.empty_like(src).pin_memory()
        lat.step_host(src, dst, 2)
    np.testing.assert_array_equal(dst.numpy(), ref)
