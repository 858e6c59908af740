"""FP32 contexts without a tiling evolve two sites per thread where nx is even,
there are no beta terms and the sites exceed one wave of warps (58368 sites), with the roundings of the one-site kernel: the
state equals the one-site kernel's bit for bit (no tolerance)."""
import numpy as np
import pytest

import ewpt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(24, 48, 51), (62, 31, 31), (48, 48, 48), (130, 21, 25), (76, 61, 90)])
@pytest.mark.parametrize("drive", [(0.0, 0.0), (0.3, 0.2)])
def test_default_context_gives_the_bits_of_one_site_per_thread(shape, drive):
    import torch

    p = ewpt.baseline_couplings(shape=shape, N=shape[0], precision=ewpt.FP32)
    y = torch.from_numpy(np.random.default_rng(3).normal(size=(36, int(np.prod(shape)))) * 0.2).cuda()
    y[0] += 1.0
    got = []
    for tile in (None, (32, 4, 0, 0)):
        with ewpt.Lattice(p) as lat:
            assert lat.tiling() == (32, 4, 0, 0)
            if tile:
                lat.set_tiling(*tile)
            out = torch.empty_like(y)
            torch.cuda.synchronize()
            lat.set_state_device(y.data_ptr())
            lat.step(5, *drive)
            lat.get_state_device(out.data_ptr())
            got.append(out)
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1])
