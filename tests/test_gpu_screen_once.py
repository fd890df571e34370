"""One-shot screening, against the oracle."""
import numpy as np
import pytest

from test_zz_no_alloc import STAT_FIELDS, crossing_groups, same

pytestmark = pytest.mark.gpu


def check(engine, oracle, st, after, alive, sz, dt, thr):
    want, ws = oracle.screen(st, after, alive, sz, 0.0, dt, threshold_km=thr)
    engine.set_screening(True, thr, 1.0, 0.01)
    try:
        got, gs = engine.screen(st, after, alive, sz, 0.0, dt)
    finally:
        engine.set_screening(True, 5.0, 1.0, 0.01)
    same(got, want)
    for f in STAT_FIELDS:
        assert gs[f] == ws[f], f
    return got


@pytest.mark.parametrize("n,dt,thr", [
    (1, 10.0, 5.0), (1025, 60.0, 20.0), (20011, 30.0, 5.0),
    (20011, 0.02, 1.0),   # cell edge near 1 km: keys too wide for the counted build, sorted instead
])
def test_one_shot_screening_equals_the_oracle(engine, oracle, ks, n, dt, thr):
    st, sz, al = ks.generate_population(900 + n, min(n, 9000), n, 20, 7200.0)
    after, alive = engine.propagate(st, al, ks.DEFAULT_EPOCH_JD, 0.0, dt, 1)
    alive[:: 7] = 0
    if n == 1:
        alive[:] = 1
    check(engine, oracle, st, after, alive, sz, dt, thr)


@pytest.mark.parametrize("per_group", [1, 30, 75])
def test_end_states_gathered_or_sent_whole(engine, oracle, ks, per_group):
    """20 000 objects, whose end states are not sent with the start states: the
    rows of up to a quarter as many pairs (30^2) are gathered on the host, for
    more (75^2) the whole arrays follow; records beyond 512 come back in a
    second copy."""
    st, sz, al = ks.generate_population(7, 20000)
    after, alive = engine.propagate(st, al, ks.DEFAULT_EPOCH_JD, 0.0, 10.0, 1)
    b, a, one, s1 = crossing_groups(per_group)[:4]
    got = check(engine, oracle, np.vstack([st, b]), np.vstack([after, a]), np.concatenate([alive, one]),
                np.concatenate([sz, s1]), 10.0, 5.0)
    assert len(got) >= per_group ** 2
