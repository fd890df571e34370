"""One-shot screening with each cell build, and the build that tests share.

The one-shot call does not say which build it took, so each is asked for:
counted (2, the default), the cooperative sort's setting (1) and the separate
kernels (0), on the same inputs, against the oracle.
"""
import numpy as np
import pytest

from test_zz_no_alloc import STAT_FIELDS, crossing_groups, same

pytestmark = pytest.mark.gpu


def screen_with(ks, form, args, dt, thr):
    with ks.Engine(0) as eng:
        eng.set_tuning("sort_fused", form)
        eng.set_screening(True, thr, 1.0, 0.01)
        # Twice: the second call finds the tables as the first one left them.
        eng.screen(*args, 0.0, dt)
        return eng.screen(*args, 0.0, dt)


@pytest.mark.parametrize("n,dt,thr", [
    (1, 10.0, 5.0), (33, 60.0, 20.0), (1025, 60.0, 20.0), (20011, 30.0, 5.0),
    (20011, 0.02, 1.0),   # cell edge near 1 km: keys too wide for the counted build, which turns to the sort
])
def test_each_build_equals_the_oracle(ks, oracle, n, dt, thr):
    st, sz, al = ks.generate_population(900 + n, min(n, 9000), n, 20, 7200.0)
    with ks.Engine(0) as eng:
        after, alive = eng.propagate(st, al, ks.DEFAULT_EPOCH_JD, 0.0, dt, 1)
    alive[::7] = 0
    if n == 1:
        alive[:] = 1
    want, ws = oracle.screen(st, after, alive, sz, 0.0, dt, threshold_km=thr)
    for form in (2, 1, 0):
        got, gs = screen_with(ks, form, (st, after, alive, sz), dt, thr)
        same(got, want)
        for f in STAT_FIELDS:
            assert gs[f] == ws[f], (form, f)


@pytest.mark.parametrize("per_group", [30, 75])
def test_each_build_with_end_states_gathered_or_sent_whole(ks, oracle, per_group):
    st, sz, al = ks.generate_population(7, 20000)
    b, a, one, s1 = crossing_groups(per_group)[:4]
    with ks.Engine(0) as eng:
        after, alive = eng.propagate(st, al, ks.DEFAULT_EPOCH_JD, 0.0, 10.0, 1)
    args = (np.vstack([st, b]), np.vstack([after, a]), np.concatenate([alive, one]), np.concatenate([sz, s1]))
    want, ws = oracle.screen(*args, 0.0, 10.0, threshold_km=5.0)
    assert len(want) >= per_group ** 2
    for form in (2, 1, 0):
        got, gs = screen_with(ks, form, args, 10.0, 5.0)
        same(got, want)
        for f in STAT_FIELDS:
            assert gs[f] == ws[f], (form, f)


def test_the_shared_engine_takes_the_default_build(engine, ks):
    """After tests that choose another build on it (this file sorts behind them)."""
    engine.set_clock(ks.DEFAULT_EPOCH_JD, 0.0, 10.0)
    engine.set_screening(True, 5.0, 1.0, 0.01)
    engine.set_population(*ks.generate_population(9, 3000))
    engine.run(2)
    engine.take_conjunctions()
    engine.take_step_stats()
    assert engine.timing()["sort_cells_fused"] == 2
