"""Calls that follow one another on one engine -- hours after a run that ended early, and after a
launch whose blocks did not find one another --, worlds at the small end of what is accepted, and
engines that share the GPU from several threads."""
import json
import threading

import numpy as np
import pytest

from helpers import COVID_FAST, make_config, rows_to_array

pytestmark = pytest.mark.gpu


def _engine(cfg, **kw):
    from epirust_gb300 import Config, Epidemiology

    return Epidemiology(Config(json.dumps(cfg)), **kw)


def _rows(r):
    return np.stack([r[k] for k in r.dtype.names], axis=1).astype(np.int64)


def _same_world(eng, sim):
    eng.check_invariants()
    assert (eng.snapshot().view(np.uint8) == sim.export().view(np.uint8)).all()


@pytest.mark.parametrize("hour_kernels", [False, True])
@pytest.mark.parametrize("n,grid", [(1500, 93), (17000, 290)])
def test_hours_after_a_run_that_ended_early(gpu, oracle_mod, n, grid, hour_kernels):
    """The run's last chain reaches into a claim window (128 hours) that its world never gets to;
    hours of that window then find no claim of the window before."""
    disease = dict(COVID_FAST, last_day=4, high_transmission_start_day=3, regular_transmission_rate=0.0,
                   high_transmission_rate=0.0)
    cfg = make_config(n=n, grid=grid, hours=193, seed=n, disease=disease, starting=(0, 0, 3, 0))
    sim = oracle_mod.O1(oracle_mod.params_from_config(cfg))
    want = rows_to_array(sim.run(1, 193, interventions=True, stop=True))
    assert 24 < len(want) < 128
    eng = _engine(cfg)
    assert (_rows(eng.run()) == want).all()
    if hour_kernels:
        eng.set_launch_shape((n + 255) // 256, 4)
    want = rows_to_array(sim.run(200, 220, interventions=False, stop=False))
    assert (_rows(eng.simulate_hours(200, 20)) == want).all()
    _same_world(eng, sim)
    eng.close()


@pytest.mark.parametrize("hour", [1, 9])
def test_a_wait_that_runs_out_ends_the_call_and_the_engine(gpu, hour):
    """A world that runs as one grid, its blocks given no time to wait for one another: the call
    reports it, the engine takes no more hours in either form, and others are not touched by it."""
    from epirust_gb300 import EpiError

    cfg = make_config(n=17000, grid=290, seed=2, disease=COVID_FAST, starting=(0, 0, 5, 50))
    want = _engine(cfg).simulate_hours(1, 24)
    eng = _engine(cfg)
    if hour > 1:
        eng.simulate_hours(1, hour - 1)
    eng.set_wait_limit(0)
    with pytest.raises(EpiError, match="TIMEOUT.*gave up waiting"):
        eng.simulate(hour)
    eng.set_wait_limit(1 << 22)
    with pytest.raises(EpiError, match="TIMEOUT"):
        eng.simulate(hour + 1)
    eng.set_launch_shape(16, 4)
    with pytest.raises(EpiError, match="TIMEOUT"):
        eng.simulate(hour + 1)
    eng.close()
    assert (_engine(cfg).simulate_hours(1, 24) == want).all()


@pytest.mark.parametrize("grid", [1, 2, 3, 5])
def test_records_of_the_smallest_grids(gpu, oracle_mod, grid):
    """Two agents at home in worlds of 4 to 36 cells: their records come back, hour after hour."""
    cfg = make_config(n=2, grid=grid, seed=9, starting=(0, 0, 0, 0))
    p = oracle_mod.params_from_config(cfg)
    recs = oracle_mod.O1(oracle_mod.params_from_config(make_config(n=2, grid=60, seed=9, starting=(0, 0, 0, 0)))).export()
    for k in (0, 1):
        for name, v in [("x", k), ("y", k), ("flags", 0), ("work_status", 3), ("work_start_at", 0), ("home_x", 0), ("home_y", 0),
                        ("work_x", 0), ("work_y", 0), ("area_x0", 0), ("area_y0", 0), ("area_x1", 1), ("area_y1", 1)]:
            recs[name][k] = v
    sim = oracle_mod.O1(p, records=recs)
    eng = _engine(cfg, records=recs)
    _same_world(eng, sim)
    want = rows_to_array(sim.run(1, 49, interventions=False, stop=False))
    assert (_rows(eng.simulate_hours(1, 48)) == want).all()
    _same_world(eng, sim)
    eng.close()


# sizes of 128, 256, 288, 512 and 544 threads a block on 152 SMs, and the longest call of one launch
@pytest.mark.parametrize("n,grid,longest", [(16_385, 330, 100), (38_912, 494, 100), (38_913, 495, 3), (77_824, 700, 3),
                                            (77_825, 700, 1), (155_648, 990, 1)])
def test_longest_call_of_one_launch(gpu, n, grid, longest):
    """Beyond it an engine would hold every SM against engines of other threads for too long."""
    eng = _engine(make_config(n=n, grid=grid, seed=3, starting=(0, 0, 0, 50)))
    hour = 1
    for k in (1, longest, min(longest + 1, 100)):
        launched = eng.kernels_launched()
        eng.simulate_hours(hour, k)
        assert (eng.kernels_launched() - launched == 1) == (k <= longest), k
        hour += k
    eng.close()


@pytest.mark.parametrize("n,grid", [(9_000, 240), (30_000, 433), (60_000, 612), (98_000, 783)])
def test_engines_of_several_threads(gpu, n, grid):
    """Four engines stepped from four threads at once, in calls of one launch and of many, have the
    hours that each has alone by hour kernels."""
    cfgs = [make_config(n=n, grid=grid, seed=70 + i, disease=COVID_FAST, starting=(0, 0, 5, 60)) for i in range(4)]
    cuts = [1, 2, 3, 6, 7, 8, 11, 14, 26, 27, 50, 73]
    got, errors = [None] * 4, []

    def work(i):
        try:
            eng = _engine(cfgs[i])
            rows = [_rows(eng.simulate_hours(a, b - a)) for a, b in zip(cuts, cuts[1:])]
            got[i] = (np.concatenate(rows), eng.snapshot())
            eng.check_invariants()
            eng.close()
        except Exception as e:  # reported below, in the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for i in range(4):
        eng = _engine(cfgs[i])
        eng.set_launch_shape((n + 255) // 256, 4)
        assert (got[i][0] == _rows(eng.simulate_hours(1, 72))).all(), i
        assert (got[i][1].view(np.uint8) == eng.snapshot().view(np.uint8)).all(), i
        eng.close()


def test_short_calls_after_the_autotuner(gpu):
    """A grid tuned on a day of hours leaves calls of an hour to the one launch that runs them, and a
    shape that is asked for does not."""
    for n, grid in [(3_000, 150), (30_000, 433), (60_000, 612), (98_000, 783), (150_000, 975)]:
        eng = _engine(make_config(n=n, grid=grid, seed=4, starting=(0, 0, 0, 50)))
        eng.autotune(24)
        launched = eng.kernels_launched()
        eng.simulate(1)
        eng.simulate(7)
        assert eng.kernels_launched() == launched + 2, n
        shape = eng.launch_shape()
        eng.set_launch_shape(**shape)
        eng.simulate(8)
        assert eng.kernels_launched() > launched + 3, n
        eng.close()


def test_algorithmic_bytes_of_an_hour(gpu):
    """The agent words and planes that the hour kernels move: 24 B an agent and 1.25 B a cell while
    people are about, and the figure that bench.py takes for one launch."""
    import bench

    n, grid = 5000, 120
    eng = _engine(make_config(n=n, grid=grid, seed=1))
    cells = (grid + 1) ** 2
    for hour in range(24, 48):
        hod = hour % 24
        want = n * 8.0 if hod == 1 else 0.0 if hod < 7 and hod else n * 20.0 if hod in (0, 23) else n * 24.0 + 1.25 * cells
        assert eng.hour_bytes(hour) == want == bench.moved_bytes(hod, n, grid), hod
    assert eng.hour_bytes(9) == bench.DECIDE_BYTES_PER_AGENT * n + bench.DECIDE_PLANES * cells
    eng.close()
