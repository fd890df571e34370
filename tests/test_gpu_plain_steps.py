"""Runs without screening, many steps to a launch, at the edges of its chunks (128 steps, two in flight)."""
import numpy as np
import pytest

from test_gpu_parity import run_engine

pytestmark = pytest.mark.gpu


def falling_population(ks, n):
    """A catalogue in which some objects re-enter within minutes of each other and some are dead from the start."""
    st, sz, al = ks.generate_population(77 + n, n)
    rng = np.random.default_rng(n)
    down = rng.choice(n, max(1, n // 6), replace=False)
    r = np.linalg.norm(st[down, :3], axis=1, keepdims=True)
    st[down, :3] *= (6378.137 + rng.uniform(20.0, 3000.0, (len(down), 1))) / r
    st[down, 3:] = -3.0 * st[down, :3] / np.linalg.norm(st[down, :3], axis=1, keepdims=True)
    al[rng.choice(n, n // 9, replace=False)] = 0
    return st, sz, al


@pytest.mark.parametrize("n,steps", [(1, 1), (31, 127), (129, 128), (1000, 129), (5003, 259), (257, 384)])
def test_plain_steps_equal_the_oracle(engine, oracle, ks, n, steps):
    st, sz, al = falling_population(ks, n)
    want = oracle.run(st, sz, al, steps=steps, screen=False)
    fs, fa = engine.propagate(st, al, ks.DEFAULT_EPOCH_JD, 0.0, 10.0, steps)
    assert np.array_equal(fs, want[0]) and np.array_equal(fa, want[1])
    # The same through a resident population, in two runs, with its counters.
    engine.set_clock(ks.DEFAULT_EPOCH_JD, 0.0, 10.0)
    engine.set_screening(False)
    try:
        engine.set_population(st, sz, al)
        for k in (steps // 3, steps - steps // 3):
            engine.run(k)
        fs, fa = engine.get_population()
        stats = engine.take_step_stats()
        assert engine.clock()[1] == steps
    finally:
        engine.set_screening(True, 5.0, 1.0, 0.01)
    assert np.array_equal(fs, want[0]) and np.array_equal(fa, want[1])
    assert np.array_equal(stats["step"], np.arange(steps))
    # The oracle counts nothing without screening: each step's count from its states up to that step.
    for k in {1, min(steps, 128), steps}:
        assert stats["alive"][k - 1] == oracle.run(st, sz, al, steps=k, screen=False)[1].sum()


def test_split_plain_steps_equal_single_steps(engine, ks):
    """Split precision: many steps to a launch against one (per-phase timing launches them singly)."""
    st, sz, al = falling_population(ks, 3001)
    out = []
    engine.set_precision(ks.PRECISION_SPLIT)
    engine.set_screening(False)
    try:
        for profiling in (False, True):
            engine.set_profiling(profiling)
            engine.set_clock(ks.DEFAULT_EPOCH_JD, 0.0, 10.0)
            engine.set_population(st, sz, al)
            engine.run(200)
            out.append((*engine.get_population(), engine.take_step_stats()["alive"]))
    finally:
        engine.set_profiling(False)
        engine.set_screening(True, 5.0, 1.0, 0.01)
        engine.set_precision(ks.PRECISION_FP64)
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_screened_run_after_a_plain_run(engine, oracle, ks):
    """Screening switched on between runs starts from the states the plain run left."""
    st, sz, al = ks.generate_population(502, 4000, 12000, 8, 3600.0)
    engine.set_clock(ks.DEFAULT_EPOCH_JD, 0.0, 10.0)
    engine.set_screening(False)
    try:
        engine.set_population(st, sz, al)
        engine.run(5)
    finally:
        engine.set_screening(True, 5.0, 1.0, 0.01)
    engine.run(3)
    fs, fa = engine.get_population()
    conj = engine.take_conjunctions()
    engine.take_step_stats()
    want = oracle.run(st, sz, al, steps=8)
    late = want[2][want[2]["step"] >= 5]
    assert np.array_equal(fs, want[0]) and np.array_equal(fa, want[1])
    assert len(conj) == len(late)
    for f in ("i", "j", "t", "miss_km", "collision"):
        assert np.array_equal(conj[f], late[f]), f
