"""The surrogate's row and gradient kernels at the edges of their tiles: any
number of rows, raw rows standardised on the device, batch sizes that take each
split of the weight gradients."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(max_batch, seed=3):
    from emt6ro.surrogate import Surrogate
    return Surrogate(max_batch=max_batch, seed=seed)


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 640, 1000])
def test_rows_of_any_count_match_the_oracle(n):
    from oracle import mlp_oracle as mo
    net = _net(128)
    x = np.random.default_rng(n).normal(size=(n, 100)).astype(np.float32)
    y, _ = mo.mixed_forward(net.get_params(), x)
    got = net.predict_std(x)
    # the forward bound of the whole-network test: 0.5% (L2) of the BF16 oracle
    assert got.shape == (n,)
    assert np.linalg.norm(got - y) <= 5e-3 * np.linalg.norm(y)
    # a row's value does not depend on its place in a tile
    assert np.array_equal(net.predict_std(x[-1:]), got[-1:])


def test_raw_rows_are_standardised_as_numpy_does():
    net = _net(256)
    rng = np.random.default_rng(8)
    x = (rng.normal(size=(777, 100)) * 40 + 5).astype(np.float32)
    net.x_mean = rng.normal(size=100).astype(np.float32)
    net.x_std = rng.uniform(0.1, 9, 100).astype(np.float32)
    net.y_mean, net.y_std = 3.0, 2.0
    want = net.predict_std((x - net.x_mean) / net.x_std).astype(np.float64) * 2.0 + 3.0
    assert np.array_equal(net.predict(x), want)
    assert np.array_equal(net.predict(x[::3]), want[::3])      # strided rows
    net.x_mean = net.x_mean.astype(np.float64)                 # standardised by numpy
    assert np.allclose(net.predict(x), want, rtol=1e-2, atol=1e-2)


def test_not_a_number_reaches_its_row_only():
    net = _net(128)
    x = np.random.default_rng(2).normal(size=(130, 100)).astype(np.float32)
    y = net.predict_std(x)
    x[5, 7], x[129, 0] = np.nan, np.inf
    z = net.predict_std(x)
    assert np.isnan(z[5]) and not np.isfinite(z[129])
    keep = np.setdiff1d(np.arange(130), [5, 129])
    assert np.array_equal(y[keep], z[keep])


@pytest.mark.parametrize("n", [4608, 4609, 5001, 19_999])
def test_more_rows_than_run_at_once(n):
    """Clusters that go over several tiles of rows give what short calls do."""
    net = _net(128)
    rng = np.random.default_rng(n)
    x = (rng.normal(size=(n, 100)) * 3).astype(np.float32)
    net.x_mean = rng.normal(size=100).astype(np.float32)
    net.x_std = rng.uniform(0.5, 2, 100).astype(np.float32)
    y = net.predict(x)
    assert np.array_equal(y, np.concatenate([net.predict(x[i:i + 999]) for i in range(0, n, 999)]))


def test_rows_in_pieces_on_the_device():
    net = _net(128)
    x = np.random.default_rng(4).normal(size=(1000, 100)).astype(np.float32)
    y = net.predict_std(x)
    net._PIECE = 333
    assert np.array_equal(net.predict_std(x), y) and np.array_equal(net.predict_std(x[:0]), y[:0])


# 128 and 384 rows: one part; 640: two; 1024: four; 2048: eight
@pytest.mark.parametrize("batch", [128, 384, 640, 1024, 2048])
def test_gradients_and_step_at_every_split(batch):
    from oracle import mlp_oracle as mo
    net = _net(2048, seed=batch)
    rng = np.random.default_rng(batch)
    x = rng.normal(size=(batch, 100)).astype(np.float32)
    t = rng.normal(size=batch).astype(np.float32)
    before = net.get_params()
    got, loss = net.gradients(x, t)
    want, want_loss = mo.mixed_gradients(before, x, t)
    assert loss == pytest.approx(want_loss, rel=5e-3)
    for k, (g, w) in enumerate(zip(got, want)):
        # the gradient bound of the whole-network test: 3% (L2) of the BF16 oracle
        assert np.linalg.norm(g - w) <= 0.03 * np.linalg.norm(w), k
    net.train_step(x, t, 1e-3)
    zeros = [np.zeros_like(p) for p in before]
    # Adam on the kernel's own gradients, in FP32 on the host
    step, _, _ = mo.adam(before, got, zeros, [z.copy() for z in zeros], 1, 1e-3)
    for k, (a, b) in enumerate(zip(net.get_params(), step)):
        assert np.allclose(a, b, rtol=0, atol=2e-6), k


def test_losses_of_consecutive_steps_do_not_mix():
    """Each step reports its own batch's loss, whether or not the one before was read."""
    from emt6ro import _native as N
    import torch
    net = _net(128)
    rng = np.random.default_rng(1)
    x = rng.normal(size=(128, 100)).astype(np.float32)
    t = rng.normal(size=128).astype(np.float32)
    want = net.train_step(x, t, 0.0)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    torch.cuda.synchronize()
    loss = ctypes.c_float()
    for read in (False, True, True, False, False, True):
        N.check(N.lib().emt6_mlp_train_step(net._h, xd.data_ptr(), td.data_ptr(), 128, 0.0,
                                            ctypes.byref(loss) if read else None))
        if read:
            assert loss.value == pytest.approx(want, rel=1e-5)


def _stall(net, phase, us=200):
    from emt6ro import _native as N
    N.check(N.lib().emt6_test_mlp_stall(net._h, phase, us))


@pytest.mark.parametrize("phase", range(6))
@pytest.mark.parametrize("batch", [128, 1024])
def test_a_wait_that_runs_out_in_training_is_reported(batch, phase):
    """The first CTA's issuer gives up in each phase of the row kernel and in the
    gradient kernel: the cluster still goes through every exchange and returns, the
    step reports the error, and the same work on another handle is right."""
    from emt6ro import _native as N
    rng = np.random.default_rng(batch)
    x = rng.normal(size=(batch, 100)).astype(np.float32)
    t = rng.normal(size=batch).astype(np.float32)
    net = _net(1024)
    want, _ = net.gradients(x, t)
    _stall(net, phase)
    with pytest.raises(N.NativeError, match="timed out"):
        net.train_step(x, t, 1e-3)
    got, _ = _net(1024).gradients(x, t)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n,phase", [(1, 0), (200, 1), (30_000, 2)])
def test_a_wait_that_runs_out_in_scoring_is_reported(n, phase):
    """Predictions of a launch that gave up are not returned."""
    from emt6ro import _native as N
    net = _net(128)
    x = np.random.default_rng(n).normal(size=(n, 100)).astype(np.float32)
    want = net.predict(x)
    _stall(net, phase)
    with pytest.raises(N.NativeError, match="timed out"):
        net.predict(x)
    _stall(net, phase)
    with pytest.raises(N.NativeError, match="timed out"):
        net.predict_std(x)
    assert np.array_equal(_net(128).predict(x), want)


@pytest.mark.parametrize("batch", [128, 640, 1024, 2048])
@pytest.mark.parametrize("phase", [0, 4, 5])
def test_a_failed_step_leaves_weights_alone(batch, phase):
    """A step whose rows failed updates nothing; one whose first gradient CTA
    failed (a part of W3's first tile) leaves that tile as it was.  Reading the
    parameters of such a handle reports the error."""
    from emt6ro import _native as N
    rng = np.random.default_rng(batch)
    x = rng.normal(size=(batch, 100)).astype(np.float32)
    t = rng.normal(size=batch).astype(np.float32)
    net = _net(2048)
    before = net.get_params()
    _stall(net, phase)
    xd, td = net._to_dev(x), net._to_dev(t)
    N.check(N.lib().emt6_mlp_train_step(net._h, xd.data_ptr(), td.data_ptr(), batch, 1e-3, None))
    after = [np.zeros_like(p) for p in before]
    rc = N.lib().emt6_mlp_get_params(net._h, (ctypes.c_void_p * 8)(*[a.ctypes.data for a in after]))
    assert rc == N.EMT6_ERR_DEVICE
    if phase == 5:
        assert np.array_equal(after[4][:128, :128], before[4][:128, :128])
        assert not np.array_equal(after[4], before[4])
    else:
        for a, b in zip(after, before):
            assert np.array_equal(a, b)


def test_each_step_reports_its_own_batchs_loss():
    """Batches of different losses in turn, some steps' losses unread: what is read
    is the loss of that step's batch, not of the one before or of a sum."""
    from emt6ro import _native as N
    net = _net(128)
    rng = np.random.default_rng(5)
    x = rng.normal(size=(128, 100)).astype(np.float32)
    batches, want = [], []
    for k in range(3):
        t = ((k + 1) ** 2 * rng.normal(size=128)).astype(np.float32)
        want.append(_net(128).train_step(x, t, 0.0))
        batches.append((net._to_dev(x), net._to_dev(t)))
    assert want[0] < 0.5 * want[1] < 0.25 * want[2]
    loss = ctypes.c_float()
    for k, read in zip([0, 1, 2, 0, 2, 1, 1, 0, 2, 2, 0], [1, 1, 0, 1, 1, 0, 1, 0, 0, 1, 1]):
        xd, td = batches[k]
        N.check(N.lib().emt6_mlp_train_step(net._h, xd.data_ptr(), td.data_ptr(), 128, 0.0,
                                            ctypes.byref(loss) if read else None))
        if read:
            assert loss.value == pytest.approx(want[k], rel=1e-5)
