"""FP64 stencils in integer arithmetic (csrc/fixstencil.cuh) against exact
rational arithmetic, through the drop-in rates: with g' = 0 and a constant
Higgs field kt_Y_i = lap Y_i - d_i Sigma and k_Sigma = (1 - gp2) d_i E^Y_i.

Bound per site, M the largest magnitude in the stencil: an aligned value is
off by less than one unit of 2^-55 M, which the weights turn into at most
1794 units (Laplacian, over 180 dx^2) and 55 units (derivative, over 60 dx);
the weighed Laplacian drops at most 64 units more, a divergence 4; then come
the rounding of the sum and of the few operations after it, 8 x 2^-53 of
their terms."""
from fractions import Fraction as Fr

import numpy as np
import pytest

import ewpt

pytestmark = pytest.mark.gpu

DX = 0.25
U = 2.0 ** -53


@pytest.fixture(scope="module", autouse=True)
def built():
    import build_lib

    build_lib.build()


def rates(shape, y):
    import torch

    p = ewpt.baseline_couplings(shape=shape, N=shape[0], dx=DX, gy=0.0)
    d = torch.from_numpy(y).cuda()
    out = torch.zeros_like(d)
    torch.cuda.synchronize()
    ewpt.rk4_rates_device(p, [d[a].data_ptr() for a in range(36)], [out[a].data_ptr() for a in range(36)],
                          stream=torch.cuda.current_stream().cuda_stream)
    return p, out.cpu().numpy()


def fields(shape, kind, seed):
    rng = np.random.default_rng(seed)
    S = int(np.prod(shape))
    y = np.zeros((36, S))
    y[0] = 1.0
    for a in (13, 14, 15, 19, 33, 34, 35):
        if kind == "random":
            v = rng.normal(size=S)
        elif kind == "smooth":
            k, j, i = np.meshgrid(*(np.arange(n) for n in shape[::-1]), indexing="ij")
            v = 0.97 + 0.3 * np.sin(2 * np.pi * i / shape[0] + a) * np.cos(2 * np.pi * (j / shape[1] - k / shape[2]))
            v = v.ravel() + 1e-3 * rng.normal(size=S)
        elif kind == "wide":  # neighbours up to 2^120 apart, zeros among them
            v = rng.normal(size=S) * 2.0 ** rng.integers(-60, 60, S)
            v[rng.random(S) < 0.2] = 0.0
        else:  # a few sites in a lattice of zeros
            v = np.where(rng.random(S) < 0.02, rng.normal(size=S), 0.0)
        y[a] = v
    return y


def exact(f, shape, axes):
    """Exact 60 dx d_axis f for each axis, 180 dx^2 lap f and the largest
    magnitude of the stencil, per site."""
    nx, ny, nz = shape
    F = np.array([Fr(float(v)) for v in f], dtype=object).reshape(nz, ny, nx)

    def r(k, ax):
        return np.roll(F, -k, axis=2 - ax)

    g = [45 * (r(1, a) - r(-1, a)) - 9 * (r(2, a) - r(-2, a)) + (r(3, a) - r(-3, a)) for a in axes]
    lap = sum(w * (r(k, a) + r(-k, a) - 2 * F) for a in range(3) for k, w in ((1, 270), (2, -27), (3, 2)))
    A = np.abs(f).reshape(nz, ny, nx)
    m = A.copy()
    for a in range(3):
        for k in (-3, -2, -1, 1, 2, 3):
            m = np.maximum(m, np.roll(A, k, axis=2 - a))
    return [v.ravel() for v in g], lap.ravel(), m.ravel()


@pytest.mark.parametrize("kind", ["random", "smooth", "wide", "sparse"])
@pytest.mark.parametrize("shape", [(7, 8, 9), (34, 7, 7)])
def test_rates_of_the_stencils(shape, kind):
    y = fields(shape, kind, 3)
    p, out = rates(shape, y)
    (gS), _, mS = exact(y[19], shape, (0, 1, 2))
    err2 = fp2 = 0.0
    for i in range(3):
        _, lap, mY = exact(y[13 + i], shape, ())
        ref = np.array([l / Fr(180 * DX * DX) - g / Fr(60 * DX) for l, g in zip(lap, gS[i])])
        terms = np.array([abs(l) / Fr(180 * DX * DX) + abs(g) / Fr(60 * DX) for l, g in zip(lap, gS[i])], dtype=float)
        bound = (1794 + 64) * U / 4 * mY / (180 * DX * DX) + 55 * U / 4 * mS / (60 * DX) + 8 * U * terms
        err = np.array([abs(Fr(float(v)) - w) for v, w in zip(out[33 + i], ref)], dtype=float)
        assert (err <= bound).all()
        err2 += (err ** 2).sum()
        fp2 += (np.array([abs(Fr(float(v)) - w) for v, w in zip(float_rate(y, shape, i), ref)], dtype=float) ** 2).sum()
    assert err2 <= fp2  # no further off than the sum in FP64
    gE = [exact(y[33 + i], shape, (i,)) for i in range(3)]
    w = Fr(1.0 - p.gp2)
    ref = [w * (a + b + c) / Fr(60 * DX) for a, b, c in zip(*(g[0][0] for g in gE))]
    mE = np.maximum.reduce([g[2] for g in gE])
    bound = float(w) * ((3 * 55 + 12) * U / 4 * mE / (60 * DX)) + 8 * U * np.array([abs(v) for v in ref], dtype=float)
    assert (np.array([abs(Fr(float(v)) - r) for v, r in zip(out[19], ref)], dtype=float) <= bound).all()


def float_rate(y, shape, i):
    """lap Y_i - d_i Sigma in FP64, weights as FP64 numbers."""
    nx, ny, nz = shape
    Y, S = y[13 + i].reshape(nz, ny, nx), y[19].reshape(nz, ny, nx)
    lap = 3.0 * (-49.0 / 18.0) * Y
    for k, w in ((1, 1.5), (2, -0.15), (3, 1.0 / 90.0)):
        lap = lap + w * sum(np.roll(Y, s * k, axis=a) for a in range(3) for s in (-1, 1))
    g = sum(w * (np.roll(S, -k, axis=2 - i) - np.roll(S, k, axis=2 - i)) for k, w in ((1, 45.0), (2, -9.0), (3, 1.0)))
    return (lap / (DX * DX) - g / (60.0 * DX)).ravel()


@pytest.mark.parametrize("special", [np.inf, np.nan, 5e-324, 1e-300, 1e300])
def test_values_outside_the_integer_range(special):
    """Infinities, NaN, denormals and magnitudes near the ends of the range
    take the floating-point evaluation: the same sites as in NumPy's are
    finite, and those are within its rounding of the exact value (at most 16
    roundings, those of the weights among them, of terms that add up to 3264
    times the largest magnitude over 180 dx^2 and 110 times over 60 dx)."""
    shape = (9, 8, 7)
    S = int(np.prod(shape))
    y = np.zeros((36, S))
    y[0] = 1.0
    y[13:16] = y[19] = 1.0
    if np.isfinite(special) and special < 1e-200:
        y[13:16] = y[19] = 0.0
    y[13:16, 100] = special
    y[19, 17] = special
    _, out = rates(shape, y)
    fin = np.where(np.isfinite(y), y, 0.0)
    for i in range(3):
        with np.errstate(all="ignore"):
            ok = np.isfinite(float_rate(y, shape, i))
        assert (np.isfinite(out[33 + i]) == ok).all()
        g, _, mS = exact(fin[19], shape, (i,))
        _, lap, mY = exact(fin[13 + i], shape, ())
        for q in np.flatnonzero(ok):
            ref = lap[q] / Fr(180 * DX * DX) - g[0][q] / Fr(60 * DX)
            bound = 16 * U * (3264 * mY[q] / (180 * DX * DX) + 110 * mS[q] / (60 * DX)) + 64 * 5e-324
            assert abs(Fr(float(out[33 + i][q])) - ref) <= Fr(bound)


@pytest.mark.parametrize("shape", [(24, 20, 28), (75, 31, 34), (75, 61, 90), (64, 64, 64), (33, 7, 9)])
@pytest.mark.parametrize("beta", [0.0, 0.3])
def test_picked_shape_gives_the_bits_of_the_default_tile(shape, beta):
    """A tile set by ewpt_set_tiling changes no bit of the FP64 form (its
    6th-order stages run four warps per 32 sites whatever the tile)."""
    import torch

    p = ewpt.baseline_couplings(shape=shape, N=shape[0], beta_w=beta)
    y = torch.randn(36, int(np.prod(shape)), dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(5)) * 0.1
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
            lat.step(3)
            lat.get_state_device(out.data_ptr())
            got.append(out)
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1])
