"""Device memory that runs out, made on the host ("deny_alloc": the n-th
allocation reports that there is none).

The second set of step buffers is held for speed alone: without room for it
steps run in one stream, and an allocation that fails while it is held takes
it back. Results never change.
"""
import numpy as np
import pytest

from conftest import golden_path
from test_gpu_breakup import EVENT_FIELDS
from test_gpu_parity import STAT_FIELDS, assert_same_conj, assert_same_stats

pytestmark = pytest.mark.gpu


def configured(ks, spg=32, dt=10.0):
    eng = ks.Engine(0)
    eng.set_steps_per_graph(spg)
    eng.set_clock(ks.DEFAULT_EPOCH_JD, 0.0, dt)
    eng.set_screening(True, 5.0, 1.0, 0.01)
    return eng


def holds_second(ks, eng):
    """Whether the second set is held (a failing allocation is then repeated without it). Gives it back."""
    eng.set_tuning("deny_alloc", 1)
    try:
        eng.set_l2_flush(1 << 20)
    except ks.KsError:
        return False
    eng.set_l2_flush(0)
    return True


def results(eng):
    return (*eng.get_population(), eng.take_conjunctions(), eng.take_step_stats())


def same(got, want):
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert_same_conj(got[2], want[2])
    assert_same_stats(got[3], want[3])


@pytest.fixture(scope="module")
def crowd(ks, oracle):
    st, sz, al = ks.generate_population(505, 5000, 30000, 8, 3600.0)
    want = oracle.run(st, sz, al, steps=12)
    assert len(want[2]) > 10
    return (st, sz, al), want


@pytest.mark.parametrize("nth", [0, 1, 2, 3])
@pytest.mark.parametrize("spg,chunks", [(0, [5, 1, 6]), (4, [4, 4, 4]), (3, [3, 2, 3, 4])])
def test_no_room_for_the_second_set(ks, crowd, nth, spg, chunks):
    pop, want = crowd
    with configured(ks, spg) as eng:
        eng.set_population(*pop)
        eng.set_tuning("deny_alloc", nth)
        eng.prepare_run()
        for k in chunks:
            eng.run(k)
        same(results(eng), want)
        if spg:   # prepare_run does nothing without graphs
            assert holds_second(ks, eng) == (nth == 0)


@pytest.mark.parametrize("spg", [0, 4])
def test_short_runs_do_without_the_second_set(ks, crowd, spg):
    """Its allocation takes longer than a few steps gain by it: a new context
    does not make it for them, and does once they have added up."""
    pop, want = crowd
    with configured(ks, spg) as eng:
        eng.set_population(*pop)
        for k in (1, 3):
            eng.run(k)
        assert not holds_second(ks, eng)
        eng.run(8)
        same(results(eng), want)
        for _ in range(20):
            eng.run(1)
        assert holds_second(ks, eng)
    with configured(ks, spg) as eng:
        eng.set_population(*pop)
        eng.run(32)
        assert holds_second(ks, eng)


@pytest.mark.parametrize("what", ["pairs", "records"])
@pytest.mark.parametrize("nth", [1, 2])
@pytest.mark.parametrize("spg", [4, 5])
def test_lists_that_grow_in_a_replay(ks, crowd, what, nth, spg):
    """The first and the second list of pairs, or the record buffer, find no memory when a chunk's overflow grows them."""
    pop, want = crowd
    with configured(ks, spg) as eng:
        eng.set_population(*pop)
        eng.prepare_run()
        eng.set_buffer_limits(*((2, 0) if what == "pairs" else (0, 2)))
        eng.set_tuning("deny_alloc", nth)
        eng.run(12)
        same(results(eng), want)
        assert not holds_second(ks, eng)


@pytest.mark.parametrize("nth", [1, 2])
def test_items_that_grow_in_a_replay(ks, nth):
    """More work items than the list first holds (one column block each), against the sorted build."""
    st, sz, al = ks.generate_population(17, 28340, 400000, 60, 3600.0)
    runs = []
    for form in (2, 0):
        with configured(ks, 4, 20.0) as eng:
            eng.set_tuning("sort_fused", form)
            eng.set_tuning("item_col_blocks", 1)
            eng.set_population(st, sz, al)
            eng.prepare_run()
            if form == 2:
                eng.set_buffer_limits(1 << 21, 1 << 18)  # only the items overflow
                eng.set_tuning("deny_alloc", nth)
            eng.run(4)
            runs.append(results(eng))
            if form == 2:
                assert not holds_second(ks, eng)
    assert len(runs[0][2]) > 0
    same(runs[0], runs[1])


@pytest.mark.parametrize("where", ["second set", "pairs", "fragments"])
@pytest.mark.parametrize("nth", [1, 2])
@pytest.mark.parametrize("spg", [1, 2, 7])
def test_fragmentation_without_the_second_set(ks, where, nth, spg):
    """Fragmentation reads a step's start and end states: in two state buffers or three, over every chunk parity."""
    fx = dict(np.load(golden_path("run_breakup.npz")))
    idx, mass, vrel, step = fx["impact"]
    with ks.Engine(0) as eng:
        eng.set_steps_per_graph(spg)
        eng.set_clock(float(fx["epoch_jd"]), 0.0, float(fx["dt"]))
        eng.set_screening(True, float(fx["threshold_km"]), float(fx["radius_scale"]), float(fx["min_vrel_km_s"]))
        eng.set_population(fx["states"], fx["size_m"], fx["alive"])
        eng.set_masses(fx["mass_kg"])
        eng.set_breakup(True, float(fx["lc_m"]), 40.0, int(fx["seed"]))
        if where == "second set":
            eng.set_tuning("deny_alloc", nth)
        eng.prepare_run()
        if where == "pairs":
            eng.set_buffer_limits(1, 0)
            eng.set_tuning("deny_alloc", nth)
        eng.run(int(step))
        if where == "fragments":
            eng.set_tuning("deny_alloc", nth)
        eng.impact(int(idx), float(mass), float(vrel))
        eng.run(int(fx["steps"]) - int(step))
        fs, fa = eng.get_population()
        conj, events, stats = eng.take_conjunctions(), eng.take_breakups(), eng.take_step_stats()
    assert np.array_equal(fs, fx["out_states"]) and np.array_equal(fa, fx["out_alive"])
    assert_same_conj(conj, fx["out_conj"])
    for f in EVENT_FIELDS:
        assert np.array_equal(events[f], fx["out_events"][f]), f
    for f in STAT_FIELDS:
        assert np.array_equal(stats[f], fx["out_stats"][f]), f


@pytest.mark.parametrize("cut", [4, 5, 6, 7, 8])
def test_second_set_taken_back_between_a_step_and_its_fragmentation(ks, cut):
    """The first collision's parents are gathered from the step's start and end
    states into a buffer made then. Where that takes the second set back, the
    start states stay at hand: chunks of `cut` steps end with them in the third
    state buffer (5, 6) or in one of the two that remain (4, 7, 8)."""
    fx = dict(np.load(golden_path("run_breakup.npz")))
    first = 12   # step of the first collision when nothing is forced before it
    runs = []
    for nth in (0, 1):
        with ks.Engine(0) as eng:
            eng.set_steps_per_graph(32)
            eng.set_clock(float(fx["epoch_jd"]), 0.0, float(fx["dt"]))
            eng.set_screening(True, float(fx["threshold_km"]), float(fx["radius_scale"]), float(fx["min_vrel_km_s"]))
            eng.set_population(fx["states"], fx["size_m"], fx["alive"])
            eng.set_masses(fx["mass_kg"])
            eng.set_breakup(True, float(fx["lc_m"]), 40.0, int(fx["seed"]))
            eng.prepare_run()
            eng.run(first + 1 - cut)
            eng.set_tuning("deny_alloc", nth)
            eng.run(20)
            runs.append((*results(eng), eng.take_breakups()))
    assert runs[0][4]["step"][0] == first and runs[0][4]["fragments"][0] > 0
    same(runs[1], runs[0])
    for f in EVENT_FIELDS:
        assert np.array_equal(runs[1][4][f], runs[0][4][f]), f


def test_autotune_and_flush_buffer_take_the_second_set_back(ks, crowd):
    pop, want = crowd
    with configured(ks, 4) as eng:
        eng.set_population(*pop)
        eng.prepare_run()
        eng.set_tuning("deny_alloc", 1)
        eng.autotune(1)
        eng.set_tuning("cell_scale_permille", 1000)   # candidate counts are those of the reference's cells
        eng.run(12)
        got = results(eng)
    same(got, want)


def test_every_allocation_of_a_population_may_fail(ks, crowd):
    """An upload that finds no memory is an error, the next one starts afresh;
    where only the counted build's words find none, cells are sorted."""
    pop, want = crowd
    with configured(ks) as eng:
        for nth in range(1, 100):
            eng.set_tuning("deny_alloc", nth)
            try:
                eng.set_population(*pop)
                break
            except ks.KsError:
                continue
        assert nth > 20
        eng.run(12)
        assert eng.timing()["sort_cells_fused"] == 1
        same(results(eng), want)
