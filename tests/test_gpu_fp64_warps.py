"""The FP64 stages' blocks of four warps and 32 sites: every rate against the
CPU oracle where the last block holds 32, 1, 31 or few sites, with and without
the beta terms (whose Higgs parts lie in shared memory of their own).

Tolerance: 1e-12 of the array's largest rate, the FP64 parity bar; a rate is a
sum of fewer than 100 terms of 1e-1 to 1e1 of that size, each within a few 2^-53.
"""
import numpy as np
import pytest

import ewpt
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 8), (7, 7, 9), (7, 9, 17), (8, 8, 11), (33, 7, 9)])
@pytest.mark.parametrize("beta", [(0.0, 0.0), (0.3, -0.2), (0.0, 0.4)])
def test_rates_of_four_warp_blocks(shape, beta):
    import torch

    orc.build()
    p = ewpt.Params(shape=shape, N=shape[0], beta_w=beta[0], beta_y=beta[1], gp2=0.6)
    S = int(np.prod(shape))
    y = np.random.default_rng(7).normal(size=(36, S)) * 0.3
    y[0] += 1.0
    d = torch.from_numpy(y).cuda()
    out = torch.full((36, S + 32), 7.0, dtype=torch.float64, device="cuda")  # 32 sentinels behind each array
    torch.cuda.synchronize()
    ewpt.rk4_rates_device(p, [d[a].data_ptr() for a in range(36)], [out[a].data_ptr() for a in range(36)], 0.3, 0.2)
    torch.cuda.synchronize()
    assert (out[:, S:] == 7.0).all()
    r = out[:, :S].cpu().numpy()
    o = orc.params(p.dims, p.dx, p.gw, p.gy, p.gp2, p.lam, p.vev, p.beta_w, p.beta_y, p.theta_w, order=p.stencil_order)
    ref = orc.rates(o, y, 0.3, 0.2)
    scale = np.abs(ref).max(axis=1)
    assert (np.abs(r - ref).max(axis=1) <= 1e-12 * scale).all()
