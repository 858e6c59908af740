"""The integer FP64 stencils (csrc/fixstencil.cuh), compiled for the host by
oracle/devstage.cc.

Divergences and curls keep the last bits of each of their arrays, however
far apart the arrays' magnitudes are.  Bound per site: an aligned value is
off by less than one unit, 2^-55 of the largest magnitude on its line of
neighbours, which the weights turn into at most 55 units of that line; then
come the rounding of each derivative and of the sums, 4 x 2^-53 of the
terms."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from oracle import devstage  # noqa: E402

U = 2.0 ** -53


def lines(f, shape, ax):
    """60 dx d_ax f and the largest magnitude among the six neighbours, in extended precision."""
    nx, ny, nz = shape
    F = f.reshape(nz, ny, nx).astype(np.longdouble)
    d, m = 0, 0
    for k, w in ((1, 45), (2, -9), (3, 1)):
        p, q = np.roll(F, -k, axis=2 - ax), np.roll(F, k, axis=2 - ax)
        d = d + w * (p - q)
        m = np.maximum(m, np.maximum(abs(p), abs(q)))
    return d.ravel(), m.ravel()


@pytest.mark.parametrize("big", [0, 1, 2])
@pytest.mark.parametrize("eps", [1.0, 1e-3, 1e-6, 1e-10, 1e-40])
def test_divergence_and_curl_of_arrays_far_apart(big, eps):
    shape = (16, 9, 10)
    n = shape[::-1]
    rng = np.random.default_rng(4)
    x = [2 * np.pi * v / m for v, m in zip(np.meshgrid(*map(np.arange, n), indexing="ij"), n)]
    y = np.zeros((36, int(np.prod(shape))))
    for c in range(3):
        wave = np.sin(x[0] + x[1] + c) + np.cos(x[2] + x[1]) + 0.1 * rng.normal(size=n)
        y[33 + c] = 1.0 if c == big else eps * wave.ravel()
    d = [[lines(y[33 + c], shape, ax) for ax in range(3)] for c in range(3)]

    def close(got, terms):
        ref = sum(s * t[0] for s, t in terms)
        bound = sum(55 * U / 4 * t[1] + 4 * U * abs(t[0]) for _, t in terms if (t[0] != 0).any())
        return (abs(got - ref) <= bound).all()

    div = [(1, d[c][c]) for c in range(3)]
    curl = [[(1, d[(i + 2) % 3][(i + 1) % 3]), (-1, d[(i + 1) % 3][(i + 2) % 3])] for i in range(3)]
    assert close(devstage.stencils(shape, y, 33)[7], div)
    out = devstage.diffs(shape, y, 33)
    assert close(out[3], div)
    for i in range(3):
        assert close(out[4 + i], curl[i])


@pytest.mark.parametrize("kind", ["random", "wide", "zeros"])
def test_stencils_are_odd(kind):
    """Those of -y are minus those of y, bit for bit, as with IEEE sums: wherever
    the values' bits are dropped, and where zeros keep their sign."""
    shape = (11, 8, 9)
    rng = np.random.default_rng(2)
    y = rng.normal(size=(36, int(np.prod(shape))))
    if kind == "wide":
        y *= 2.0 ** rng.integers(-60, 60, y.shape)
    if kind == "zeros":
        y[rng.random(y.shape) < 0.3] = 0.0
    minus = np.where(y == 0.0, 0.0, -y)
    for f in (devstage.stencils, devstage.diffs):
        np.testing.assert_array_equal(f(shape, minus, 4), -f(shape, y, 4))
