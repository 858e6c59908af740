"""FP32-form launches laid along the rows (tiles that would leave more than an
eighth of their lanes without a site): the same bits as tiles, for rows
shorter and longer than a block, chunks of fewer rows, and one or two sites per
thread; and the shape picked without ewpt_set_tiling, too."""
import pytest

import ewpt

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build_lib

    build_lib.build()


def evolve(p, y, tile, n=3, comp=False):
    import torch

    with ewpt.Lattice(p) as lat:
        if tile:
            lat.set_tiling(*tile)
        if comp:
            lat.set_fp32_compensated(True)
        out = torch.empty_like(y)
        torch.cuda.synchronize()
        lat.set_state_device(y.data_ptr())
        lat.step(n, Jex=0.02, gamma=0.01)
        lat.get_state_device(out.data_ptr())
        return out


def state(shape, seed):
    import math

    import torch

    y = torch.randn(36, math.prod(shape), dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(seed)) * 0.1
    y[0] += 1.0
    return y


# (flat tile, tile that fits or nearly fits) per lattice
PAIRS = [((24, 34, 9), (64, 2, 2, 1), (4, 8, 2, 1)), ((74, 61, 10), (64, 2, 2, 1), (1, 32, 2, 1)),
         ((160, 32, 8), (64, 2, 2, 1), (16, 8, 2, 1)), ((8, 7, 40), (32, 4, 0, 1), (4, 8, 0, 1)),
         ((260, 33, 8), (64, 2, 2, 1), (2, 16, 2, 1))]


@pytest.mark.parametrize("shape,flat,tile", PAIRS)
@pytest.mark.parametrize("beta", [0.0, 0.2])
def test_paired_rows(shape, flat, tile, beta):
    import torch

    p = ewpt.baseline_couplings(shape=shape, N=shape[0], precision=ewpt.FP32, beta_w=beta)
    y = state(shape, 3)
    a, b = evolve(p, y, flat), evolve(p, y, tile)
    assert torch.isfinite(a).all() and torch.equal(a, b)
    if beta == 0.0:
        assert torch.equal(evolve(p, y, flat, comp=True), evolve(p, y, tile, comp=True))


@pytest.mark.parametrize("shape,flat,tile", [((75, 61, 9), (64, 2, 2, 0), (1, 32, 2, 0)),
                                             ((33, 7, 9), (32, 4, 0, 0), (1, 32, 0, 0)),
                                             ((131, 40, 7), (64, 2, 1, 0), (4, 8, 1, 0))])
def test_single_rows(shape, flat, tile):
    import torch

    p = ewpt.baseline_couplings(shape=shape, N=shape[0], precision=ewpt.FP32)
    y = state(shape, 4)
    a, b = evolve(p, y, flat), evolve(p, y, tile)
    assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("shape", [(24, 24, 24), (48, 48, 48), (64, 40, 36), (75, 61, 20)])
def test_picked_shape(shape):
    import torch

    p = ewpt.baseline_couplings(shape=shape, N=shape[0], precision=ewpt.FP32)
    y = state(shape, 5)
    assert torch.equal(evolve(p, y, None), evolve(p, y, (4, 8, 0, 0)))
