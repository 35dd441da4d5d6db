"""The selector's network where sums leave the range, where the tile kernels' scratch is refused, and its
forward pass over several tiles a CTA and odd layers."""
import numpy as np
import pytest

import atc

pytestmark = pytest.mark.gpu


def _case(B, I, H, O, seed):
    rng = np.random.default_rng(seed)
    net = atc.MLP(I, H, O, seed=seed)
    mean = rng.normal(size=I).astype(np.float32)
    std = (rng.random(I) + 0.5).astype(np.float32)
    net.scaling(mean, std)
    return net, rng.normal(size=(B, I)).astype(np.float32), rng.normal(size=(B, O)).astype(np.float32), mean, std


def _layers64(params, I, H, O, z):
    p = params.astype(np.float64)
    out, at = [], 0
    for a, b in ((I, H), (H, H), (H, O)):
        out.append((p[at:at + a * b].reshape(a, b), p[at + a * b:at + a * b + b]))
        at += a * b + b
    (w1, b1), (w2, b2), (w3, b3) = out
    a1 = np.maximum(z @ w1 + b1, 0)
    a2 = np.maximum(a1 @ w2 + b2, 0)
    return a1, a2, a2 @ w3 + b3, w2, w3


def _gradients64(params, I, H, O, z, t):
    a1, a2, y, w2, w3 = _layers64(params, I, H, O, z)
    dy = (y - t) / y.size
    d2 = (dy @ w3.T) * (a2 > 0)
    d1 = (d2 @ w2.T) * (a1 > 0)
    return np.concatenate([np.concatenate([(u.T @ v).ravel(), v.sum(0)]) for u, v in ((z, d1), (a1, d2), (a2, dy))])


@pytest.mark.parametrize("B", [1, 8, 480, 4096])
@pytest.mark.parametrize("size", [1e21, 1e30, 1e36])
def test_targets_beyond_the_loss(B, size):
    """The squared errors leave the range, so the loss is an infinity; the gradients do not.  Sums of up to
    4096 x 24 terms in FP32 against 64 bits: 2e-4 of the largest, as for ordinary targets."""
    net, x, t, mean, std = _case(B, 6, 64, 24, B)
    t = (t * np.float32(size)).astype(np.float32)
    loss, g = net.gradients(x, t)
    assert loss == np.inf
    z = (x.astype(np.float64) - mean) / std.astype(np.float64)
    want = _gradients64(net.params(), 6, 64, 24, z, t.astype(np.float64))
    assert np.abs(g - want).max() <= 2e-4 * np.abs(want).max()


def test_one_infinite_target():
    """Gradients of an infinite error: infinite or no number where it enters, never a finite value."""
    net, x, t, _, _ = _case(9, 6, 64, 24, 2)
    t[3, 5] = np.inf
    loss, g = net.gradients(x, t)
    assert loss == np.inf
    b3 = g[-24:]
    assert b3[5] == -np.inf and np.isfinite(np.delete(b3, 5)).all()


@pytest.mark.parametrize("B,H", [(30, 64), (480, 64), (480, 100)])
def test_no_room_for_the_tiles(B, H):
    """The layer kernels take over where the tile kernels' sums are refused; the values agree within the
    tolerance of both against the oracle."""
    net, x, t, _, _ = _case(B, 6, H, 24, 3)
    loss, g = net.gradients(x, t)
    p = net.params()
    # what the layers hold: rows of 6, 24 and H values several times over, and the gradients
    layers = 4 * (B * (6 + 4 * 24 + 4 * H) + p.size + 64)
    try:
        atc.set_alloc_budget(layers)
        loss2, g2 = net.gradients(x, t)
        atc.set_alloc_budget(2 * layers)
        net.train(x, t, epochs=1, batch=B, seed=1)
    finally:
        atc.set_alloc_budget(None)
    assert abs(loss - loss2) <= 1e-4 * max(1.0, abs(loss))
    assert np.abs(g - g2).max() <= 2e-4 * max(np.abs(g).max(), 1e-3)


@pytest.mark.parametrize("B", [1, 7, 8, 9, 480, 1217, 1300, 5000])
@pytest.mark.parametrize("I,H,O", [(6, 64, 24), (6, 64, 60), (3, 33, 7), (6, 100, 60), (1, 1, 1), (6, 160, 24)])
def test_forward_values(B, I, H, O):
    """Sums of up to 160 products in FP32 against 64 bits: 1e-5 of the largest output."""
    net, x, _, mean, std = _case(B, I, H, O, B + H)
    z = (x.astype(np.float64) - mean) / std.astype(np.float64)
    want = _layers64(net.params(), I, H, O, z)[2]
    got = net.forward(x)
    assert got.shape == (B, O)
    assert np.abs(got - want).max() <= 1e-5 * max(np.abs(want).max(), 1e-3)
