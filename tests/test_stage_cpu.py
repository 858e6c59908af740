"""The stage kernels' own per-site code, compiled for the host by
oracle/devstage.cc: the four warps of the 6th-order FP64 stages
(csrc/stage_fp64.cuh over the integer stencils) and the equations of the FP32
forms (csrc/physics_fp32.cuh), against the golden rates of the reference's
rk4_step! and against the oracle, to the bar of the GPU rates test."""
import os

import numpy as np
import pytest

from oracle import devstage
from oracle import oracle as orc

TOL = 1e-12  # relative to max |rate| per array


def coef(g):
    return tuple(float(g["p_" + k]) for k in ("gw", "gy", "gp2", "lambda", "vev", "beta_w", "beta_y", "dx"))


def far(r, ref):
    return float((np.abs(r - ref) / np.maximum(np.abs(ref).max(axis=1, keepdims=True), 1e-300)).max())


def state(shape, seed=11):
    y = np.random.default_rng(seed).normal(size=(36, int(np.prod(shape))))
    y[:4] += 1.0  # |Phi| away from 0 (the damping term divides by it)
    return y


@pytest.mark.parametrize("form", ["fp64", "fp32", "orders"])
@pytest.mark.parametrize("case", ["a", "b"])
def test_rates_match_golden(golden_dir, case, form):
    g = dict(np.load(os.path.join(golden_dir, f"ref_{case}.npz")))
    shape = tuple(int(v) for v in g["shape"])
    r = devstage.rates(shape, coef(g), g["y0"], float(g["Jex"]), float(g["gam"]), form)
    assert far(r, g["rates"]) < TOL


@pytest.mark.parametrize("form", ["fp64", "fp32", "orders"])
@pytest.mark.parametrize("beta", [0.0, 0.3])
@pytest.mark.parametrize("gamma", [0.0, 0.05])
def test_rates_match_oracle(form, beta, gamma):
    shape = (12, 7, 9)
    y = state(shape)
    op = orc.params(shape, 0.25, 0.65, 0.35, 0.99, 0.129, 1.0, beta, -beta)
    ref = orc.rates(op, y, 0.7, gamma)
    r = devstage.rates(shape, (0.65, 0.35, 0.99, 0.129, 1.0, beta, -beta, 0.25), y, 0.7, gamma, form)
    assert far(r, ref) < TOL


@pytest.mark.parametrize("beta", [0.0, 0.3])
def test_fp64_rates_of_minus_phi(beta):
    """Those of the Higgs arrays change sign, the others stay, to the bit."""
    shape = (8, 9, 7)
    y = state(shape, 3)
    y[2][np.random.default_rng(1).random(y.shape[1]) < 0.3] = 0.0
    sign = np.ones((36, 1))
    sign[[0, 1, 2, 3, 20, 21, 22, 23]] = -1.0
    c = (0.65, 0.35, 0.99, 0.129, 1.0, beta, -beta, 0.25)
    a = devstage.rates(shape, c, y, 0.7, 0.05)
    b = devstage.rates(shape, c, np.where(y == 0.0, 0.0, sign * y), 0.7, 0.05)
    np.testing.assert_array_equal(b, sign * a)
