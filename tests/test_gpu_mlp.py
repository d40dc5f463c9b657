"""The controller network's CUDA forward/backward/Adam kernels against the
FP64 numpy restatement (oracle/mlp_oracle.py)."""
import numpy as np
import pytest

import dsgdpp_b200 as P
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


def _net(seed=3):
    net = P.Mlp(seed=seed)
    rng = np.random.default_rng(seed)
    net.params = rng.normal(0, 0.15, net.n_params).astype(np.float32)
    return net, rng


def test_forward_matches_oracle():
    net, rng = _net()
    X = rng.normal(0, 1.5, (40, 16)).astype(np.float32)
    got = net.forward(X)
    want, _ = M.forward(net.params, X)
    np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-5)
    assert np.all(np.abs(got) <= 1.0)


def test_gradient_matches_oracle():
    net, rng = _net(5)
    X = rng.normal(0, 1.0, (64, 16)).astype(np.float32)
    y = rng.uniform(-0.9, 0.9, 64).astype(np.float32)
    loss, g = net.gradient(X, y)
    wl, wg = M.loss_and_grad(net.params, X, y)
    assert loss == pytest.approx(wl, rel=1e-4)
    scale = np.max(np.abs(wg))
    np.testing.assert_allclose(g, wg, rtol=2e-3, atol=2e-5 * scale)
    # deterministic reduction: the same call gives the same bits
    _, g2 = net.gradient(X, y)
    assert np.array_equal(g, g2)


def test_training_reduces_loss():
    net = P.Mlp(seed=11)
    rng = np.random.default_rng(2)
    X = rng.normal(0, 1, (512, 16)).astype(np.float32)
    y = (0.6 * np.tanh(X[:, 0] - 0.5 * X[:, 3])).astype(np.float32)
    first = net.train_step(X, y, lr=3e-3)
    for _ in range(300):
        last = net.train_step(X, y, lr=3e-3)
    assert last < 0.2 * first


@pytest.mark.parametrize("batch", [1, 3, 148, 149, 151, 592, 593, 1190])
def test_batches_that_fill_and_leave_samples_in_the_last_block(batch):
    # one sample per block up to 148, then four at a time; 64-term FP32 dot
    # products of values of order 1 err by some 1e-6, tolerances as above
    net, rng = _net(batch)
    X = rng.normal(0, 1.0, (batch, 16)).astype(np.float32)
    y = rng.uniform(-0.9, 0.9, batch).astype(np.float32)
    want, _ = M.forward(net.params, X)
    np.testing.assert_allclose(net.forward(X), want, rtol=1e-4, atol=1e-5)
    loss, g = net.gradient(X, y)
    wl, wg = M.loss_and_grad(net.params, X, y)
    assert loss == pytest.approx(wl, rel=1e-4)
    np.testing.assert_allclose(g, wg, rtol=2e-3, atol=2e-5 * np.max(np.abs(wg)))
    # a training step moves every parameter against its gradient, by lr at first
    before = net.params
    assert net.train_step(X, y, lr=1e-3) == loss
    moved = net.params - before
    clear = np.abs(g) > 1e-4
    np.testing.assert_allclose(moved[clear], -1e-3 * np.sign(g[clear]), rtol=1e-2)


@pytest.mark.parametrize("batch", [1, 3, 148, 149, 592, 1190])
def test_outputs_are_fp64_sums_rounded_once(batch):
    # an output of at most 1 rounds by up to 3e-8; FP32 sums of its 64 terms err
    # by more than 1e-7 in some samples of the larger batches
    net, rng = _net(batch + 1)
    X = rng.normal(0, 1.0, (batch, 16)).astype(np.float32)
    want, _ = M.forward(net.params, X)
    np.testing.assert_allclose(net.forward(X), want, rtol=0, atol=6e-8)


@pytest.mark.parametrize("batch", [1, 3, 64, 148])
def test_gradients_of_few_samples_near_their_targets(batch):
    # targets 1e-4 off the outputs: an output that errs by 1e-7 puts 1e-3 of its
    # gradient in error, the FP32 operations that follow the outputs some 1e-6
    net, rng = _net(batch + 2)
    X = rng.normal(0, 1.0, (batch, 16)).astype(np.float32)
    y = (M.forward(net.params, X)[1][-1] + 1e-4).astype(np.float32)
    want, wg = M.loss_and_grad(net.params, X, y)
    loss, g = net.gradient(X, y)
    assert loss == pytest.approx(want, rel=1e-5)
    np.testing.assert_allclose(g, wg, rtol=0, atol=1e-5 * np.max(np.abs(wg)))
