"""Device memory of a surrogate handle: the minibatches that training gathers ahead take theirs from
the first training call on, and a handle whose calls come in any order computes the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net():
    from epirust_gb300.surrogate import Surrogate

    # 64 KB of inputs a step in each orientation, 128 steps ahead: 16.8 MB beside a network of 0.5 MB
    return Surrogate(in_dim=8, hidden=128, hidden_layers=1, out_dim=6, batch=512, seed=3)


def test_only_training_holds_minibatches(gpu):
    import torch

    rng = np.random.default_rng(0)
    x, y = rng.random((2048, 8)), rng.random((2048, 6))

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    warm = _net()  # the library's own first allocations
    warm.predict(x[:10])
    warm.gradients(x[:512], y[:512])
    before = used()
    nets = [_net() for _ in range(4)]
    for net in nets:
        net.predict(x[:10])
        net.gradients(x[:512], y[:512])
    idle = used() - before
    for net in nets:
        net.set_dataset(x, y)
        net.train(128, seed=1)
    trained = used() - before
    for net in nets + [warm]:
        net.close()
    assert idle < 4 * (8 << 20)
    assert trained < 4 * (40 << 20)


def test_calls_in_any_order(gpu):
    """Training calls of growing length with gradients in between, against fresh handles."""
    rng = np.random.default_rng(1)
    x, y = rng.random((2048, 8)), rng.random((2048, 6))
    net = _net()
    net.set_dataset(x, y)
    start = net.get_params()
    for steps in (2, 4, 9, 130, 5, 261):
        fresh = _net()
        g, want_g = net.gradients(x[:512], y[:512])[1], fresh.gradients(x[:512], y[:512])[1]
        assert np.array_equal(g, want_g), steps
        fresh.set_dataset(x, y)
        want = fresh.train(steps, seed=steps)
        assert np.allclose(net.train(steps, seed=steps), want, rtol=1e-4), steps  # (losses are summed by atomics)
        assert np.array_equal(net.get_params(), fresh.get_params()), steps
        net.set_params(start)
        fresh.close()
    net.close()
