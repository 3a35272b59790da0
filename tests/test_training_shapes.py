"""The training kernels at the shapes where they can go wrong: one layer and four, the smallest
and padded outputs, batches of one to four row tiles, narrow and wide tiles (few and many
networks), step counts around the captured group and the gathered chunk, and Adam's step count
across calls."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


def _net(**kw):
    from epirust_gb300.surrogate import Surrogate

    return Surrogate(**kw)


# (in_dim, hidden, hidden_layers, out_dim, batch, members)
SHAPES = [(1, 128, 1, 1, 128, 1), (64, 128, 2, 129, 128, 13), (5, 384, 3, 130, 384, 2), (8, 512, 4, 600, 512, 7),
          (3, 256, 1, 128, 256, 40)]


@pytest.mark.parametrize("shape", SHAPES)
def test_gradients_match_oracle(gpu, shape):
    """Tolerances of the fixed-shape test: loss 1e-3, each layer's gradients 2e-2 relative
    (FP32 against float64 accumulation, and BF16 roundings that land on the other side)."""
    in_dim, hidden, depth, out, batch, members = shape
    rng = np.random.default_rng(sum(shape))
    net = _net(in_dim=in_dim, hidden=hidden, hidden_layers=depth, out_dim=out, batch=batch, members=members, seed=3)
    x, t = rng.random((batch, in_dim)), rng.random((batch, out)) * 0.5
    loss, g = net.gradients(x, t)
    loss, g, p = np.atleast_1d(loss), np.atleast_2d(g), np.atleast_2d(net.get_params())
    for m in {0, members // 2, members - 1}:
        want_loss, want = omlp.loss_and_gradients(omlp.unflatten(p[m], net.shapes), x, t, emulate=True)
        assert loss[m] == pytest.approx(want_loss, rel=1e-3)
        for l, ((gw, gb), (ww, wb)) in enumerate(zip(omlp.unflatten(g[m], net.shapes), want)):
            assert np.linalg.norm(gw - ww) / np.linalg.norm(ww) < 2e-2, (m, l)
            assert np.linalg.norm(gb - wb) / np.linalg.norm(wb) < 2e-2, (m, l)
    net.close()


@pytest.mark.parametrize("steps", [1, 3, 4, 5, 128, 133])
def test_wide_and_narrow_tiles_train_alike(gpu, steps):
    """Twelve networks (wide tiles) equal, bit for bit, networks trained alone (narrow tiles)."""
    shape = dict(in_dim=6, hidden=256, hidden_layers=2, out_dim=140, batch=256)
    rng = np.random.default_rng(steps)
    x, y = rng.random((700, 6)), rng.random((700, 140)) * 0.5
    ens = _net(members=12, seed=50, **shape)
    ens.set_dataset(x, y)
    losses, params = ens.train(steps, seed=9), ens.get_params()
    assert losses.shape == (12, steps) and np.isfinite(losses).all() and (losses > 0).all()
    for m in (0, 5, 11):
        one = _net(seed=50 + m, **shape)
        one.set_dataset(x, y)
        lo = one.train(steps, seed=9 + m)
        assert np.array_equal(one.get_params(), params[m]), m
        assert np.allclose(lo, losses[m], rtol=1e-4), m
        one.close()
    ens.close()


def test_adam_counts_steps_across_calls(gpu):
    """The third of three one-step calls on a one-minibatch set is Adam's step 3 with the moments
    of the first two, on the handle's own gradients (tolerance of the one-step test: 2e-6 where
    |g| is well above eps)."""
    rng = np.random.default_rng(8)
    net = _net(in_dim=8, hidden=256, hidden_layers=2, out_dim=100, batch=128, seed=6)
    x, t = rng.random((128, 8)), rng.random((128, 100)) * 0.5
    net.set_dataset(x, t)
    m = v = 0.0
    for step in (1, 2, 3):
        p0 = net.get_params().astype(np.float64)
        g = net.gradients(x, t)[1].astype(np.float64)
        net.train(1, seed=0)
        want, m, v = omlp.adam_step(p0, g, m, v, step, 1e-3, 0.9, 0.999, 1e-8)
        sel = np.abs(g) > 1e-6
        assert np.allclose(net.get_params().astype(np.float64)[sel], want[sel], rtol=0, atol=2e-6), step
    net.close()
