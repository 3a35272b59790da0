"""The inference products at the shapes where they can go wrong: K of one block, of the whole
resident panel and beyond it (the tile-per-CTA kernel), one column block, an odd number of them
(two at a time and a last one alone), rows that fill the SMs (whole rows per work item, several
items per CTA) and rows that do not."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu

# (in_dim, hidden, hidden_layers, out_dim, members, rows)
SHAPES = [(1, 128, 1, 1, 1, 1), (8, 512, 3, 600, 2, 12801), (64, 384, 2, 129, 3, 7000), (5, 640, 2, 300, 2, 700),
          (8, 256, 1, 100, 40, 500), (3, 896, 2, 128, 1, 20000), (8, 128, 1, 200, 3, 129)]


@pytest.mark.parametrize("shape", SHAPES)
def test_predictions_and_scores_match_oracle(gpu, shape):
    """Tolerances of the fixed-shape test: predictions 2e-3 relative (FP32 against float64
    accumulation, and BF16 roundings that land on the other side), scores 1e-3.  The first rows
    alone (another split of the same products) give the same bits."""
    from epirust_gb300.surrogate import Surrogate

    in_dim, hidden, depth, out, members, n = shape
    rng = np.random.default_rng(sum(shape))
    net = Surrogate(in_dim=in_dim, hidden=hidden, hidden_layers=depth, out_dim=out, batch=128, members=members, seed=5)
    x, target = rng.random((n, in_dim)), rng.random(out) * 0.5
    got, score = net.predict_members(x), net.score_members(x, target)
    assert got.shape == (members, n, out) and score.shape == (members, n)
    rows = np.unique(np.r_[0, n - 1, rng.integers(0, n, 60)])
    p = np.atleast_2d(net.get_params())
    for m in {0, members // 2, members - 1}:
        want, _ = omlp.forward(omlp.unflatten(p[m], net.shapes), x[rows], emulate=True)
        assert np.linalg.norm(got[m, rows] - want) / np.linalg.norm(want) < 2e-3, m
    exact = ((got.astype(np.float64) - target.astype(np.float32)) ** 2).sum(axis=2)
    assert np.allclose(score, exact, rtol=1e-3, atol=1e-6)
    few = min(n, 130)
    assert np.array_equal(net.predict_members(x[:few]), got[:, :few])
    net.close()
