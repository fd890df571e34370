"""Dense populations: cells sorted again once a step has shown how many pairs it holds.

140 000 objects at steps of 120 s hold some 0.85e9 candidate pairs a step
(the bounds are 0.6e9 with the second set of buffers, 0.7e9 in one stream). Only
the order in which pairs are looked at changes, so records, counters and states
equal those of the separate sort kernels, across the change from one build to
the other and back.
"""
import numpy as np
import pytest

from test_gpu_breakup import EVENT_FIELDS
from test_gpu_memory import configured, results, same

pytestmark = pytest.mark.gpu

DENSE_PAIRS = 0.7e9


@pytest.fixture(scope="module")
def dense(ks):
    return ks.generate_population(41, 28340, 140_000, 60, 86400.0)


def run(ks, pop, form, spg, chunks, setup=lambda eng: None):
    with configured(ks, spg, 120.0) as eng:
        eng.set_tuning("sort_fused", form)
        setup(eng)
        eng.set_population(*pop)
        forms = []
        for k in chunks:
            eng.run(k)
            forms.append(eng.timing()["sort_cells_fused"])
        return results(eng), forms, eng.take_breakups()


@pytest.mark.parametrize("spg,chunks", [(0, [1, 2, 5]), (3, [8]), (2, [2, 6]), (4, [40])])
def test_dense_steps_are_sorted_and_equal_the_sort_kernels(ks, dense, spg, chunks):
    got, forms, _ = run(ks, dense, 2, spg, chunks)
    want, _, _ = run(ks, dense, 0, spg, [sum(chunks)])
    assert want[3]["candidate_pairs"].min() > DENSE_PAIRS
    assert forms[-1] == 1 and (chunks[0] > 1 or forms[0] == 2)   # the first step, of unknown density, is counted
    same(got, want)


def test_builds_change_with_the_step_length(ks, dense):
    """Long steps, short ones and long ones again; screened in between, one-shot, with the counted build."""
    got = []
    for form in (2, 0):
        with configured(ks, 4, 120.0) as eng:
            eng.set_tuning("sort_fused", form)
            eng.set_population(*dense)
            out, forms = [], []
            for dt, steps in ((120.0, 5), (10.0, 40), (120.0, 5)):
                eng.set_clock(ks.DEFAULT_EPOCH_JD, eng.clock()[0], dt)
                eng.run(steps)
                forms.append(eng.timing()["sort_cells_fused"])
                out.append(results(eng))
            assert forms == ([1, 2, 1] if form == 2 else [0, 0, 0])
            got.append(out)
    for a, b in zip(*got):
        same(a, b)


@pytest.mark.parametrize("device", [False, True])
def test_dense_steps_with_fragmentation(ks, dense, device):
    """Collisions fragmented on the host (start states in three buffers, then two) and on the device (one stream)."""
    def setup(eng):
        eng.set_screening(True, 5.0, 60.0, 0.01)
        if device:
            eng.set_breakup_mode(ks.BREAKUP_DEVICE, 400_000)
        eng.set_breakup(True, 0.5, 40.0, 7)

    got, forms, events = run(ks, dense, 2, 4, [1, 9], setup)
    want, _, want_events = run(ks, dense, 0, 4, [10], setup)
    assert forms[-1] == 1
    assert len(want_events) > 0 and want[3]["candidate_pairs"].min() > DENSE_PAIRS
    same(got, want)
    for f in EVENT_FIELDS:
        assert np.array_equal(events[f], want_events[f]), f


@pytest.mark.parametrize("n,dt,chunks,form", [
    (270_000, 120.0, [1, 7], 1),    # crowded cells could be put in order by then: 4 500 pairs an object decide
    (2_000_000, 25.0, [1, 3], 0),   # too many for the cooperative sort: the separate kernels
])
def test_dense_steps_of_larger_populations(ks, n, dt, chunks, form):
    st, sz, al = ks.generate_population(43, 28340, n, 200, 86400.0)
    got = []
    for fused in (2, 0):
        with configured(ks, 3, dt) as eng:
            eng.set_precision(ks.PRECISION_SPLIT)
            eng.set_tuning("sort_fused", fused)
            eng.set_population(st, sz, al)
            for k in chunks:
                eng.run(k)
            assert eng.timing()["sort_cells_fused"] == (form if fused == 2 else 0)
            got.append(results(eng))
    assert got[1][3]["candidate_pairs"].min() > (4500 if form else 2000) * n
    same(*got)
