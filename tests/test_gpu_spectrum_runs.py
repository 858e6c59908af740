"""Log-shell binning in runs of modes along x: mode counts exactly, and sums
to 1e-11 of NumPy's for rows that are shorter than a run, whole runs and one
over, and with more shells than a row has modes (1e-11: two FFTs in FP64 and a
sum of at most 1e4 positive terms, some 1e3 roundings of 1.1e-16 at most)."""
import math

import numpy as np
import pytest

import ewpt

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build_lib

    build_lib.build()


def reference(fields, shape, nbins):
    nx, ny, nz = shape
    nmax = min(shape) // 2
    ks = [np.where(np.arange(n) <= n // 2, np.arange(n), np.arange(n) - n) for n in (nz, ny, nx)]
    m = ks[0][:, None, None] ** 2 + ks[1][None, :, None] ** 2 + ks[2][None, None, :] ** 2
    P = sum(np.abs(np.fft.fftn(f.reshape(nz, ny, nx))) ** 2 for f in fields)
    sums, counts = np.zeros(nbins), np.zeros(nbins)
    edges = np.exp(math.log(nmax) * np.arange(nbins + 1) / nbins)
    n = np.sqrt(m)
    for b in range(nbins):
        hi = (n <= nmax) if b == nbins - 1 else (n < edges[b + 1])
        sel = (m > 0) & (n >= (edges[b] if b else 0)) & hi
        sums[b], counts[b] = P[sel].sum(), sel.sum()
    return sums, counts


@pytest.mark.parametrize("shape", [(7, 8, 9), (14, 10, 12), (16, 16, 16), (30, 16, 20), (33, 18, 11)])
@pytest.mark.parametrize("nbins", [1, 6, 40, 256])
@pytest.mark.parametrize("form", [ewpt.FP64, ewpt.FP32, ewpt.DF64])
def test_shells(shape, nbins, form):
    p = ewpt.baseline_couplings(shape=shape, N=shape[0], precision=form)
    rng = np.random.default_rng(sum(shape))
    y = rng.normal(size=(36, p.sites)) * 0.1
    y[0] += 1.0
    with ewpt.Lattice(p) as lat:
        lat.set_state(y)
        for field in ("higgs", "B"):
            s = lat.spectrum(field, "log", nbins)
            sums, counts = reference(lat.fields(field), shape, nbins)
            np.testing.assert_array_equal(s["count"], counts)
            np.testing.assert_allclose(s["sum"], sums, rtol=1e-11, atol=0)
