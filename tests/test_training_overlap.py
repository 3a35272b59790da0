"""The launches of a training step overlap: each is resident while the ones before it still write
what it will read.  Whatever the timing, the same steps from the same weights give the same
weights, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,hidden,batch,members", [(1, 128, 128, 1), (3, 512, 256, 1), (2, 256, 512, 3), (4, 128, 128, 5)])
def test_training_repeats_itself(gpu, depth, hidden, batch, members):
    from epirust_gb300.surrogate import Surrogate

    rng = np.random.default_rng(depth)
    net = Surrogate(in_dim=8, hidden=hidden, hidden_layers=depth, out_dim=150, batch=batch, members=members, seed=1)
    net.set_dataset(rng.random((4 * batch, 8)), rng.random((4 * batch, 150)) * 0.5)
    start = net.get_params()
    first = None
    for _ in range(6):
        net.set_params(start)
        net.train(61, seed=2)
        got = net.get_params()
        first = got if first is None else first
        assert np.array_equal(first, got)
    assert not np.array_equal(first, start)
    net.close()
