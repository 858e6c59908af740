"""State conversions of the FP32 and DF64 forms (hi = fl32(v), lo = fl32(v -
hi), read back as hi + lo): bit for bit what NumPy's casts give, over the
whole FP64 exponent range and at the rounding ties, from host and device
memory and over rows that do not fill a block."""
import ctypes as C

import numpy as np
import pytest

import ewpt

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build_lib

    build_lib.build()


def values(shape, seed):
    rng = np.random.default_rng(seed)
    n = 36 * int(np.prod(shape))
    m = rng.integers(0, 2 ** 52, n, dtype=np.uint64)
    k = rng.integers(0, 8, n)
    tie = np.uint64(1) << np.uint64(28)
    low = np.uint64(2 ** 29 - 1)
    m = np.where(k == 0, (m & ~low) | tie, m)              # ties
    m = np.where(k == 1, (m & ~low) | (tie - np.uint64(1)), m)
    m = np.where(k == 2, (m & ~low) | (tie + np.uint64(1)), m)
    m = np.where(k == 3, m & ~low, m)                      # lo = 0
    m = np.where(k == 4, m | ~low & np.uint64(2 ** 52 - 1), m)  # carries into the exponent
    e = np.where(rng.random(n) < 0.5, rng.integers(1000, 1040, n), rng.integers(0, 1151, n)).astype(np.uint64)
    edge = rng.integers(0, 40, n)
    for q, v in enumerate((948, 949, 950, 1148, 1149, 1150)):
        e = np.where(edge == q, np.uint64(v), e)
    s = rng.integers(0, 2, n, dtype=np.uint64)
    y = ((s << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)
    y[rng.random(n) < 0.05] = 0.0
    y[rng.random(n) < 0.01] = -0.0
    return y.reshape(36, -1)


def bits(a):
    """Bit patterns, every NaN as one (its sign and payload are not defined)."""
    return np.where(np.isnan(a), np.uint64(0x7FF8 << 48), a.view(np.uint64))


@pytest.mark.parametrize("form", [ewpt.FP32, ewpt.DF64])
@pytest.mark.parametrize("shape", [(7, 7, 7), (33, 9, 11), (70, 64, 8), (66, 62, 30)])
def test_split_and_join_are_the_casts(form, shape):
    import torch

    y = values(shape, 1 + shape[0])
    with np.errstate(over="ignore", invalid="ignore", under="ignore"):
        hi = y.astype(np.float32)
        ref = hi.astype(np.float64) + (y - hi.astype(np.float64)).astype(np.float32).astype(np.float64)
    p = ewpt.baseline_couplings(shape=shape, N=shape[0], precision=form)
    with ewpt.Lattice(p) as lat:
        lat.set_state(y)
        np.testing.assert_array_equal(bits(lat.get_state()), bits(ref))
        d = torch.from_numpy(y).cuda()
        out = torch.zeros_like(d)
        torch.cuda.synchronize()
        lat.set_state_device(d.data_ptr())
        lat.get_state_device(out.data_ptr())
        np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(ref))
        # device arrays that do not lie back to back
        ptr = [d[a].data_ptr() for a in reversed(range(36))]
        lat.L.ewpt_set_state.argtypes = lat.L.ewpt_get_state.argtypes = [C.c_void_p, C.c_void_p, C.c_int32]
        assert lat.L.ewpt_set_state(lat.h, (C.c_void_p * 36)(*ptr), 1) == 0
        assert lat.L.ewpt_get_state(lat.h, (C.c_void_p * 36)(*[out[a].data_ptr() for a in range(36)]), 1) == 0
        np.testing.assert_array_equal(bits(out.cpu().numpy()[::-1]), bits(ref))


def test_ensemble_device_states():
    import torch

    shape = (18, 7, 9)
    y = values(shape, 5)
    p = ewpt.baseline_couplings(shape=shape, N=shape[0], precision=ewpt.FP32)
    with ewpt.Ensemble([p, p]) as ens:
        d = torch.from_numpy(y).cuda()
        out = torch.zeros_like(d)
        torch.cuda.synchronize()
        assert ens.L.ewpt_ensemble_set_state(ens.h, 1, d.data_ptr(), 1) == 0
        assert ens.L.ewpt_ensemble_get_state(ens.h, 1, out.data_ptr(), 1) == 0
        ens.set_state(0, y)
        np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(ens.get_state(0)))
        np.testing.assert_array_equal(bits(ens.get_state(1)), bits(ens.get_state(0)))


@pytest.mark.parametrize("form", [ewpt.FP32, ewpt.DF64, "ensemble"])
def test_a_state_past_the_end_of_its_memory_is_refused(form):
    """An error before anything is queued, and the context stays usable."""
    import torch

    from ewpt import _lib

    shape = (64, 48, 48)
    n = int(np.prod(shape))
    p = ewpt.baseline_couplings(shape=shape, N=64, precision=ewpt.FP32 if form == "ensemble" else form)
    y = torch.randn(36, n, dtype=torch.float64, device="cuda")
    cu = C.CDLL("libcuda.so.1")
    half, base, size = C.c_uint64(), C.c_uint64(), C.c_size_t()
    assert cu.cuMemAlloc_v2(C.byref(half), C.c_size_t(18 * n * 8)) == 0
    try:
        end = half.value  # of the allocations that lie back to back
        while cu.cuMemGetAddressRange_v2(C.byref(base), C.byref(size), C.c_uint64(end)) == 0:
            end = base.value + size.value
        short = end - 18 * n * 8
        torch.cuda.synchronize()
        lat = ewpt.Ensemble([p]) if form == "ensemble" else ewpt.Lattice(p)
        with lat:
            if form == "ensemble":
                def put(ptr):
                    return lat.L.ewpt_ensemble_set_state(lat.h, 0, C.c_void_p(ptr), 1)

                def get(ptr):
                    return lat.L.ewpt_ensemble_get_state(lat.h, 0, C.c_void_p(ptr), 1)
            else:
                def put(ptr):
                    return lat.L.ewpt_set_state_packed(lat.h, C.c_void_p(ptr), 1)

                def get(ptr):
                    return lat.L.ewpt_get_state_packed(lat.h, C.c_void_p(ptr), 1)
            assert put(y.data_ptr()) == 0
            assert put(short) == _lib.ERR_CUDA
            assert get(short) == _lib.ERR_CUDA
            out = torch.zeros_like(y)
            torch.cuda.synchronize()
            assert get(out.data_ptr()) == 0
            assert torch.allclose(out, y, rtol=1e-13, atol=0)
    finally:
        cu.cuMemFree_v2(half)
