"""The surrogate network's layer kernels (csrc/mlp_layers.cuh) at the edges
of their tiles and of the sizes they take, next to the general path beyond
them: forward and gradients against the FP64 oracle with the bars of
test_gpu_mlp.py (2e-3 and 2e-2, set by bfloat16 rounding flips), one AdamW step
against its formula, and the weight images after training against those
of a net that is given the trained parameters."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build_lib

    build_lib.build()


def make(dims, max_batch, seed=1):
    from ewpt.surrogate import MLP

    n_in, width, n_out = dims
    return MLP(n_in, width, n_out, max_batch=max_batch, seed=seed)


def data(dims, B, seed):
    rng = np.random.default_rng(seed)
    return (rng.normal(size=(B, dims[0])).astype(np.float32), rng.normal(size=(B, dims[2])).astype(np.float32))


# the surrogate; one feature; smallest and largest tiles; sizes past the
# layer kernels' (width no multiple of 16, n_in, n_out)
DIMS = [(84, 256, 40), (1, 32, 1), (16, 64, 32), (17, 96, 33), (130, 160, 128), (512, 512, 5), (84, 40, 40),
        (513, 64, 8), (20, 64, 129)]


def sizes(dims):
    n_in, width, n_out = dims
    return [width * n_in, width, width * width, width, n_out * width, n_out]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("B", [1, 16, 129])
def test_forward_and_gradients(dims, B):
    net = make(dims, 300)
    x, y = data(dims, B, B)
    p = net.get_params()
    f = mo.forward(p.astype(np.float64), x.astype(np.float64), *dims)
    got = net.forward(x)
    assert np.linalg.norm(got - f["z3"]) / np.linalg.norm(f["z3"]) < 2e-3
    g, loss = net.gradients(x, y)
    gr, lr_ = mo.gradients(p.astype(np.float64), x.astype(np.float64), y.astype(np.float64), *dims)
    assert abs(loss - lr_) < 1e-3 * lr_
    o = 0
    for n in sizes(dims):
        assert np.linalg.norm(g[o:o + n] - gr[o:o + n]) <= 2e-2 * np.linalg.norm(gr[o:o + n])
        o += n
    assert np.array_equal(net.get_params(), p)  # gradients leave the parameters alone
    net.close()


@pytest.mark.parametrize("dims,B", [((84, 256, 40), 128), ((17, 96, 33), 37), ((84, 256, 40), 512), ((84, 40, 40), 40),
                                    ((84, 256, 40), 600)])
def test_train_step_is_adamw_and_keeps_the_images(dims, B):
    net = make(dims, 600)
    x, y = data(dims, B, 7)
    p, m, v = net.get_params(), 0.0, 0.0
    lr, wd = 2e-3, 1e-2
    for t in range(1, 4):
        g, loss = net.gradients(x, y)
        assert abs(net.train_step(x, y, lr, wd) - loss) <= 1e-6 * loss
        m = 0.9 * m + 0.1 * g.astype(np.float64)
        v = 0.999 * v + 0.001 * g.astype(np.float64) ** 2
        step = (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8) + wd * p
        q = net.get_params()
        # FP32 arithmetic: a few roundings of the step (relative 1e-7 each, 1e-4
        # where 1 - 0.999^t cancels) and one of the parameter
        np.testing.assert_allclose(q, p - lr * step, rtol=3e-7, atol=2e-4 * lr)
        p = q.astype(np.float64)
    fresh = make(dims, 600, seed=5)
    fresh.set_params(net.get_params())
    xs, ys = data(dims, 65, 9)
    np.testing.assert_array_equal(net.forward(xs), fresh.forward(xs))
    np.testing.assert_array_equal(net.gradients(xs, ys)[0], fresh.gradients(xs, ys)[0])
    net.close()
    fresh.close()


def test_a_wait_that_runs_out_leaves_the_weights_alone():
    from ewpt import _lib

    dims = (84, 256, 40)
    net = make(dims, 128)
    x, y = data(dims, 128, 3)
    p = net.get_params()
    net.set_wait_limit(0)
    for call in (lambda: net.train_step(x, y, 1e-3), lambda: net.gradients(x, y), lambda: net.forward(x)):
        with pytest.raises(_lib.EwptError) as ei:
            call()
        assert ei.value.code == _lib.ERR_TIMEOUT
    net.set_wait_limit(-1)
    assert np.array_equal(net.get_params(), p)
    f = mo.forward(p.astype(np.float64), x.astype(np.float64), *dims)["z3"]
    assert np.linalg.norm(net.forward(x) - f) / np.linalg.norm(f) < 2e-3
    net.close()


@pytest.mark.parametrize("dims,B", [((84, 256, 40), 128), ((17, 96, 33), 37), ((84, 40, 40), 40), ((84, 256, 40), 600)])
@pytest.mark.parametrize("last", [False, True])
def test_a_step_whose_wait_runs_out_is_not_taken(dims, B, last):
    """Neither where the first kernel gives up nor where only the weight
    gradients' does (last; networks with layer kernels): parameters, moments
    and the step count are as before, so the net then trains as a fresh one
    does, bit for bit."""
    from ewpt import _lib

    layers = dims[1] % 16 == 0 and B <= 512
    if last and not layers:
        pytest.skip("no layer kernels")
    net, fresh = make(dims, 600), make(dims, 600)
    x, y = data(dims, B, 3)
    p = net.get_params()
    limit = net.L.ewpt_mlp_set_weight_wait_limit if last else net.L.ewpt_mlp_set_wait_limit
    assert limit(net.h, 0) == 0
    for _ in range(3):
        with pytest.raises(_lib.EwptError) as ei:
            net.train_step(x, y, 1e-3, 1e-2)
        assert ei.value.code == _lib.ERR_TIMEOUT
        assert np.array_equal(net.get_params(), p)
    assert limit(net.h, -1) == 0
    for _ in range(2):
        assert net.train_step(x, y, 1e-3, 1e-2) == fresh.train_step(x, y, 1e-3, 1e-2)
        assert np.array_equal(net.get_params(), fresh.get_params())
    assert np.array_equal(net.forward(x), fresh.forward(x))
    net.close()
    fresh.close()


@pytest.mark.parametrize("dims", [(84, 256, 40), (512, 512, 128)])
def test_inputs_of_any_batch(dims):
    """Around the batch from which the inputs are copied to the device first
    (393,216 floats read for all column tiles): a row's outputs do not depend
    on the batch, and a step is that of the rows' gradients."""
    rows = 393216 // (dims[0] * (dims[1] // 16))
    net = make(dims, 3000)
    x, y = data(dims, 3000, 4)
    ref = net.forward(x)
    for B in (rows - 1, rows, rows + 1, 513):
        np.testing.assert_array_equal(net.forward(x[:B]), ref[:B])
    p = net.get_params()
    for B in (rows, rows + 1):
        g, _ = net.gradients(x[:B], y[:B])
        gr, _ = mo.gradients(p.astype(np.float64), x[:B].astype(np.float64), y[:B].astype(np.float64), *dims)
        assert np.linalg.norm(g - gr) <= 2e-2 * np.linalg.norm(gr)
    net.close()


def test_a_large_batch_is_no_slower_than_on_the_general_path():
    """131072 rows: less time than a network of the next wider size that the
    layer kernels do not take (0.7 of it; 2.5 with the inputs read from host
    memory once per column tile)."""
    import time

    B, best = 131072, []
    for dims in ((84, 256, 40), (84, 264, 40)):
        net = make(dims, B)
        x, _ = data(dims, B, 5)
        net.forward(x)
        times = []
        for _ in range(5):
            t0 = time.perf_counter()
            net.forward(x)
            times.append(time.perf_counter() - t0)
        best.append(min(times))
        net.close()
    assert best[0] < 1.2 * best[1]
