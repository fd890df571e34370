"""The cell build by counting (the default), at the sizes where it can go wrong.

Cells are opened in a hash by the objects themselves, their objects placed in
arrival order, sparse cells screened by the kernel that looks up their
neighbours and the others handed to the tile kernel: records and counters must
equal the oracle's (FP64 precision: every value bit for bit) whatever the
order of arrival, and those of the sorted builds.
"""
import numpy as np
import pytest

from test_gpu_parity import assert_same_conj, assert_same_stats, run_engine

pytestmark = pytest.mark.gpu


def cluster(rng, n, spread_km):
    """n objects around one point of a circular orbit, speeds within 20 m/s: pairs inside one or a few cells."""
    st = np.zeros((n, 6))
    st[:, :3] = np.array([7000.0, 300.0, -200.0]) + rng.normal(0.0, spread_km, (n, 3))
    st[:, 3:] = np.array([0.0, 5.0, 5.6]) + rng.normal(0.0, 0.02, (n, 3))
    return st


def population(ks, kind, n):
    rng = np.random.default_rng(n)
    if kind == "catalogue":
        st, sz, al = ks.generate_population(n, n)
    elif kind == "cluster":    # one crowded cell and its neighbours
        st, sz, al = cluster(rng, n, 60.0), rng.uniform(0.1, 5.0, n), np.ones(n, np.uint8)
    else:                      # both, with dead objects in between
        st, sz, al = ks.generate_population(n, n)
        m = n // 3
        st[rng.choice(n, m, replace=False)] = cluster(rng, m, 25.0)
        al[rng.choice(n, n // 5, replace=False)] = 0
    return st, sz, al


@pytest.mark.parametrize("kind,n,dt,sub", [
    ("catalogue", 1, 10.0, 1), ("cluster", 2, 10.0, 1), ("cluster", 8, 10.0, 1),     # 28 pairs: still a sparse cell
    ("cluster", 9, 10.0, 0), ("cluster", 33, 10.0, 1), ("cluster", 700, 10.0, 3),    # around the tile kernel's 32 rows
    ("mixed", 127, 60.0, 1), ("mixed", 1025, 30.0, 2), ("mixed", 9001, 10.0, 1),
    ("catalogue", 20011, 60.0, 1),
])
def test_counted_cells_equal_the_oracle(engine, oracle, ks, kind, n, dt, sub):
    st, sz, al = population(ks, kind, n)
    engine.set_tuning("subcell_bits", sub)
    engine.set_tuning("sort_fused", 2)
    try:
        got = run_engine(engine, st, sz, al, 4, dt=dt, spg=2)
        assert engine.timing()["sort_cells_fused"] == 2
    finally:
        engine.set_tuning("subcell_bits", 1)
    want = oracle.run(st, sz, al, steps=4, dt=dt)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert_same_conj(got[2], want[2])
    assert_same_stats(got[3], want[3])


@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_counted_cells_equal_the_sorted_builds(engine, ks, precision):
    """A population with clouds, all three builds in turn on one context: each
    leaves the shared hash and counters as the next one needs them."""
    st, sz, al = ks.generate_population(31, 20000, 300000, 40, 7200.0)
    engine.set_precision(ks.PRECISION_SPLIT if precision == "split" else ks.PRECISION_FP64)
    runs = []
    try:
        for form in (2, 1, 2, 0, 2):
            engine.set_tuning("sort_fused", form)
            runs.append(run_engine(engine, st, sz, al, 5, spg=3))
            assert engine.timing()["sort_cells_fused"] == form
    finally:
        engine.set_tuning("sort_fused", 2)
        engine.set_precision(ks.PRECISION_FP64)
    assert len(runs[0][2]) > 0
    for other in runs[1:]:
        assert np.array_equal(other[0], runs[0][0]) and np.array_equal(other[1], runs[0][1])
        assert_same_conj(other[2], runs[0][2])
        assert_same_stats(other[3], runs[0][3])


@pytest.mark.parametrize("spg,chunks", [(0, [1, 2, 3, 4, 5, 6]), (4, [4, 4, 1, 4, 4, 4]), (5, [5, 5, 5, 2, 5])])
def test_refinement_beside_the_next_step(engine, oracle, ks, spg, chunks):
    """Steps whose refinement runs on a second stream while the next step
    overwrites buffers, over chunks of every parity, with records in every step."""
    st, sz, al = ks.generate_population(505, 5000, 30000, 8, 3600.0)
    got = run_engine(engine, st, sz, al, sum(chunks), spg=spg, chunks=chunks)
    want = oracle.run(st, sz, al, steps=sum(chunks))
    assert len(want[2]) > 20
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert_same_conj(got[2], want[2])
    assert_same_stats(got[3], want[3])


def test_refinement_beside_the_next_step_at_larger_sizes(engine, ks):
    """The sizes at which the propagation shares the cell build's stream and
    has one of its own again, against the sorted build in one stream."""
    for n in (140_000, 530_000):
        st, sz, al = ks.generate_population(n, 20000, n, 40, 7200.0)
        runs = []
        try:
            for form in (2, 1):
                engine.set_tuning("sort_fused", form)
                runs.append(run_engine(engine, st, sz, al, 11, spg=4))
        finally:
            engine.set_tuning("sort_fused", 2)
        assert len(runs[0][2]) > 0
        assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
        assert_same_conj(runs[0][2], runs[1][2])
        assert_same_stats(runs[0][3], runs[1][3])
