"""DF64 with two sites per thread (csrc/dd2.cuh; even rows, no beta terms,
lattices above 116,736 sites) against the FP64 form: 1e-11 of each array's
largest value after 10 steps, the form's bar, for the shortest even rows, rows
around a block's width, every register variant and a drive; and next to the
one-site kernel at the size where it takes over."""
import math

import pytest

import ewpt

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build_lib

    build_lib.build()


def state(shape, seed):
    import torch

    y = torch.randn(36, math.prod(shape), dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(seed)) * 0.1
    y[0] += 1.0
    y[30] = 0.0  # exact zeros among the momenta
    return y


def evolve(shape, form, y, tile=None, steps=10):
    import torch

    p = ewpt.baseline_couplings(shape=shape, N=shape[0], precision=form)
    with ewpt.Lattice(p) as lat:
        if tile:
            lat.set_tiling(*tile)
        out = torch.empty_like(y)
        torch.cuda.synchronize()
        lat.set_state_device(y.data_ptr())
        lat.step(steps, Jex=0.02, gamma=0.01)
        lat.get_state_device(out.data_ptr())
        return out


@pytest.mark.parametrize("shape", [(8, 121, 121), (10, 109, 108), (64, 48, 40), (130, 30, 31), (300, 57, 7),
                                   (48, 48, 50), (48, 48, 51), (49, 48, 51)])
def test_matches_fp64(shape):
    y = state(shape, 1)
    a, b = evolve(shape, ewpt.DF64, y), evolve(shape, ewpt.FP64, y)
    err = ((a - b).abs().amax(dim=1) / b.abs().amax(dim=1)).max()
    assert float(err) < 1e-11


@pytest.mark.parametrize("tile", [(32, 4, 0, 0), (64, 2, 1, 0), (16, 8, 2, 0)])
def test_register_variants_agree(tile):
    import torch

    shape = (64, 48, 40)
    y = state(shape, 2)
    assert torch.equal(evolve(shape, ewpt.DF64, y, steps=3), evolve(shape, ewpt.DF64, y, tile, steps=3))


@pytest.mark.parametrize("shape", [(50, 50, 50), (64, 48, 40)])
def test_bubbles_match_fp64(shape):
    """From a start in which most arrays are zero, and set by the device
    initialiser, whose conversion is in place."""
    import torch

    p = ewpt.baseline_couplings(shape=shape, N=shape[0])
    R, w = ewpt.ic.tanh_profile_params(p.lam, p.vev)
    bubbles = ewpt.ic.tanh_bubble_list(shape, p.dx, 4, seed=3)
    got = []
    for form in (ewpt.DF64, ewpt.FP64):
        with ewpt.Lattice(ewpt.baseline_couplings(shape=shape, N=shape[0], precision=form)) as lat:
            lat.init_bubbles(bubbles, "tanh", R, w)
            start = torch.from_numpy(lat.get_state())
            lat.step(10, Jex=0.0, gamma=0.0)
            got.append((start, torch.from_numpy(lat.get_state())))
    assert torch.all((got[0][0] - got[1][0]).abs() <= 2.0 ** -47 * got[1][0].abs())
    top = got[1][1].abs().amax(dim=1)
    err = (got[0][1] - got[1][1]).abs().amax(dim=1)
    assert torch.all(err <= 1e-11 * top)
    assert (top > 0).sum() > 20
