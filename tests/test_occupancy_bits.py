"""The hour kernels' bit planes and claim lists at the sizes where they can go wrong: rows that
end on, just before and just after a 32-bit word, dense worlds (many displaced claims), agent
counts around the 256-agent chunk, and chains that start from either buffer.  Whole numbers:
counts, every agent record and the engine's own invariants must match the CPU oracle exactly."""
import json

import numpy as np
import pytest

from helpers import COVID_FAST, make_config, rows_to_array

pytestmark = pytest.mark.gpu


def _engine(cfg):
    from epirust_gb300 import Config, Epidemiology

    return Epidemiology(Config(json.dumps(cfg)))


def _rows(r):
    return np.stack([r[k] for k in r.dtype.names], axis=1).astype(np.int64)


def _same_world(eng, sim):
    eng.check_invariants()
    assert (eng.snapshot().view(np.uint8) == sim.export().view(np.uint8)).all()


# G + 3 cells a row: one word short of a boundary, on it, one cell past it
@pytest.mark.parametrize("grid,n", [(60, 700), (61, 255), (62, 256), (92, 1700), (93, 257), (94, 2700), (125, 3000),
                                    (126, 4000)])
def test_row_words_and_dense_claims(gpu, oracle_mod, grid, n):
    cfg = make_config(n=n, grid=grid, seed=grid * 7 + n, disease=COVID_FAST, starting=(4, 4, 4, 12), beds=0.01)
    sim = oracle_mod.O1(oracle_mod.params_from_config(cfg))
    want = rows_to_array(sim.run(1, 58, interventions=False, stop=False))
    eng = _engine(cfg)
    assert (_rows(eng.simulate_hours(1, 57)) == want).all()
    _same_world(eng, sim)
    eng.close()


@pytest.mark.parametrize("cuts", [(7, 8, 9, 22, 23, 24, 31), (1, 12, 13, 16, 17, 40, 47), tuple(range(1, 30))])
def test_chains_from_either_buffer(gpu, oracle_mod, cuts):
    """Chains cut at hours of both parities, and hours run again after a restore."""
    cfg = make_config(n=1500, grid=93, seed=5, disease=COVID_FAST, starting=(2, 2, 4, 20))
    eng = _engine(cfg)
    eng.simulate_hours(1, 8)
    eng.save_state()
    for _ in range(2):
        first = 9
        sim = oracle_mod.O1(oracle_mod.params_from_config(cfg))
        sim.run(1, 9, interventions=False, stop=False)
        for cut in [c for c in cuts if c > 9] + [60]:
            want = rows_to_array(sim.run(first, cut, interventions=False, stop=False))
            assert (_rows(eng.simulate_hours(first, cut - first)) == want).all(), (first, cut)
            _same_world(eng, sim)
            first = cut
        eng.restore_state()
    eng.close()


def test_replicates_that_end_early_keep_their_buffers(gpu):
    """Replicates whose runs stop at different hours sit in different buffers; a second run from
    there, and a restore, still equal lone engines."""
    from epirust_gb300 import Config, Ensemble

    cfgs = [make_config(n=400 + 211 * i, grid=70 + 13 * i, hours=24 * 9 - 5 * i, seed=90 + i, disease=COVID_FAST,
                        starting=(1 if i % 2 else 0, 0, 1, i)) for i in range(5)]
    ens = Ensemble([Config(json.dumps(c)).params for c in cfgs])
    ens.save_state()
    lone = [_engine(c) for c in cfgs]
    for again in range(2):
        rows = ens.run()
        ens.check_invariants()
        for r, eng in enumerate(lone):
            assert (_rows(rows[r]) == _rows(eng.run())).all(), (again, r)
            assert (ens.snapshot(r).view(np.uint8) == eng.snapshot().view(np.uint8)).all(), (again, r)
    ens.restore_state()
    ens.check_invariants()
    rows = ens.run()
    for r, c in enumerate(cfgs):
        eng = _engine(c)
        assert (_rows(rows[r]) == _rows(eng.run())).all(), r
        eng.close()
    for eng in lone:
        eng.close()
    ens.close()
