"""The hour kernels' bit planes and claim lists at the sizes where they can go wrong: rows that
end on, just before and just after a 32-bit word, dense worlds (many displaced claims), agent
counts around the 256-agent chunk, and chains that start from either buffer.  Whole numbers:
counts, every agent record and the engine's own invariants must match the CPU oracle exactly."""
import json

import numpy as np
import pytest

from helpers import COVID_FAST, make_config, rows_to_array

pytestmark = pytest.mark.gpu


def _engine(cfg, hour_kernels=False):
    """An engine of a small world runs its hours in one cluster; asked for a launch shape, with
    the hour kernels of larger worlds."""
    from epirust_gb300 import Config, Epidemiology

    eng = Epidemiology(Config(json.dumps(cfg)))
    if hour_kernels:
        eng.set_launch_shape(max(1, (eng.population() + 255) // 256 - 1), 4)
    return eng


def _rows(r):
    return np.stack([r[k] for k in r.dtype.names], axis=1).astype(np.int64)


def _same_world(eng, sim):
    eng.check_invariants()
    assert (eng.snapshot().view(np.uint8) == sim.export().view(np.uint8)).all()


# G + 3 cells a row: one word short of a boundary, on it, one cell past it
@pytest.mark.parametrize("hour_kernels", [False, True])
@pytest.mark.parametrize("grid,n", [(60, 700), (61, 255), (62, 256), (92, 1700), (93, 257), (94, 2700), (125, 3000),
                                    (126, 4000)])
def test_row_words_and_dense_claims(gpu, oracle_mod, grid, n, hour_kernels):
    cfg = make_config(n=n, grid=grid, seed=grid * 7 + n, disease=COVID_FAST, starting=(4, 4, 4, 12), beds=0.01)
    sim = oracle_mod.O1(oracle_mod.params_from_config(cfg))
    want = rows_to_array(sim.run(1, 58, interventions=False, stop=False))
    eng = _engine(cfg, hour_kernels)
    assert (_rows(eng.simulate_hours(1, 57)) == want).all()
    _same_world(eng, sim)
    eng.close()


@pytest.mark.parametrize("hour_kernels", [False, True])
@pytest.mark.parametrize("cuts", [(7, 8, 9, 22, 23, 24, 31), (1, 12, 13, 16, 17, 40, 47), tuple(range(1, 30))])
def test_chains_from_either_buffer(gpu, oracle_mod, cuts, hour_kernels):
    """Chains cut at hours of both parities, and hours run again after a restore."""
    cfg = make_config(n=1500, grid=93, seed=5, disease=COVID_FAST, starting=(2, 2, 4, 20))
    eng = _engine(cfg, hour_kernels)
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


@pytest.mark.parametrize("n,grid", [(33, 60), (4096, 128), (16383, 260), (16384, 257), (16385, 261)])
def test_one_cluster_equals_hour_kernels(gpu, n, grid):
    """The run loop (lockdown, vaccination, hospital build, early stop) of the smallest and the
    largest worlds that one cluster runs, and of one agent more, against the hour kernels; the
    two also take over from each other in mid-run."""
    cfg = make_config(n=n, grid=grid, hours=24 * 40, seed=n, disease=COVID_FAST, starting=(0, 0, 1, 3 + n // 500),
                      beds=0.002, occupancy=0.5,
                      interventions=[{"Lockdown": {"at_number_of_infections": 1 + n // 100, "essential_workers_population": 0.2}},
                                     {"Vaccinate": {"at_hour": 300, "percent": 0.2}}])
    one, other = _engine(cfg), _engine(cfg, hour_kernels=True)
    one.save_state()
    want = _rows(other.run())
    assert (_rows(one.run()) == want).all()
    assert (one.snapshot().view(np.uint8) == other.snapshot().view(np.uint8)).all()
    one.check_invariants()
    if n <= 16384:
        assert one.kernels_launched() < other.kernels_launched() // 4
    one.restore_state()
    got, going = one.run_until(200)
    one.set_launch_shape(1, 4)
    if going:
        got, going = one.run_until(333)
    if going:
        got = one.run()
    assert (_rows(got) == want).all()
    assert (one.snapshot().view(np.uint8) == other.snapshot().view(np.uint8)).all()
    one.check_invariants()
    one.close()
    other.close()


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


@pytest.mark.parametrize("n,grid", [(16385, 280), (38912, 420), (38913, 421), (155648, 800), (155649, 800)])
def test_one_grid_equals_hour_kernels(gpu, n, grid):
    """The smallest and the largest worlds whose hours one grid runs (for calls of a few hours, and
    up to 38,912 agents for all), and one agent more, against the hour kernels, in calls of one to
    thirty hours over a boundary of the claim keys' window (128 hours), taking over from each
    other in between."""
    cfg = make_config(n=n, grid=grid, hours=24 * 9, seed=n, disease=COVID_FAST, starting=(0, 0, 1, 3 + n // 300), beds=0.002)
    one, other = _engine(cfg), _engine(cfg, hour_kernels=True)
    hour = 1
    for k in (1, 1, 5, 1, 1, 12, 30, 13, 11, 30, 1, 24, 2, 12):
        if hour in (53, 77):
            one.set_launch_shape(2, 4)  # from here on the hour kernels
        assert (_rows(one.simulate_hours(hour, k)) == _rows(other.simulate_hours(hour, k))).all(), hour
        hour += k
    assert hour > 130
    assert (one.snapshot().view(np.uint8) == other.snapshot().view(np.uint8)).all()
    one.check_invariants()
    one.close()
    other.close()


@pytest.mark.parametrize("n,grid", [(16385, 261), (30000, 430)])
def test_one_grid_runs_the_run_loop(gpu, n, grid):
    """Lockdown, vaccination, hospital build and the early stop, as the hour kernels have them."""
    cfg = make_config(n=n, grid=grid, hours=24 * 40, seed=n, disease=COVID_FAST, starting=(0, 0, 1, 3 + n // 500),
                      beds=0.002, occupancy=0.5,
                      interventions=[{"Lockdown": {"at_number_of_infections": 1 + n // 100, "essential_workers_population": 0.2}},
                                     {"Vaccinate": {"at_hour": 300, "percent": 0.2}}])
    one, other = _engine(cfg), _engine(cfg, hour_kernels=True)
    assert (_rows(one.run()) == _rows(other.run())).all()
    assert (one.snapshot().view(np.uint8) == other.snapshot().view(np.uint8)).all()
    one.check_invariants()
    assert one.kernels_launched() < other.kernels_launched() // 4
    one.close()
    other.close()


# chunks a block takes at a time on 152 SMs: 1, 3, 5, 9 (the last a group of 9 with one block's cut short)
@pytest.mark.parametrize("replicates,n", [(3, 700), (40, 13000), (70, 16500), (80, 24100)])
def test_replicates_in_groups_of_chunks_equal_lone_engines(gpu, replicates, n):
    from epirust_gb300 import Config, Ensemble

    cfgs = [make_config(n=n - 97 * (i % 5), grid=int((n / 0.2) ** 0.5) + i % 3, hours=40, seed=7 + i, disease=COVID_FAST,
                        starting=(0, 0, n // 100, n // 50)) for i in range(replicates)]
    ens = Ensemble([Config(json.dumps(c)).params for c in cfgs])
    rows = ens.run()
    ens.check_invariants()
    for r in (0, replicates // 2, replicates - 1):
        eng = _engine(cfgs[r], hour_kernels=True)
        assert (_rows(rows[r]) == _rows(eng.run())).all(), r
        assert (ens.snapshot(r).view(np.uint8) == eng.snapshot().view(np.uint8)).all(), r
        eng.close()
    ens.close()
