"""Crowded cells put in the order of their sub-cells (counted cell build,
populations above 262 144 objects): only the tile kernel's reading order
changes, so records, counters and states equal those of the sorted build."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_conj, assert_same_stats, run_engine

pytestmark = pytest.mark.gpu


def crowds(ks, sizes, n):
    """A thin population (0.4 km cells would hold one object each) with crowds of the given sizes, some across cell borders."""
    st, sz, al = ks.generate_population(n, 20000, n, 300, 86400.0)
    rng = np.random.default_rng(n)
    at = rng.permutation(n)
    first = 0
    for k, m in enumerate(sizes):
        rows = at[first:first + m]
        first += m
        a = 0.7 * k
        r, u = 6900.0 + 37.0 * k, np.array([np.cos(a), np.sin(a), 0.0])
        w = np.array([-np.sin(a) * 0.6, np.cos(a) * 0.6, 0.8])
        st[rows, :3] = r * u + rng.normal(0.0, 12.0 + 10.0 * (k % 3), (m, 3))
        st[rows, 3:] = 7.5 * w + rng.normal(0.0, 0.02, (m, 3))
        al[rows[::17]] = 0
    return st, sz, al


@pytest.mark.parametrize("precision,sub,spg,dt,thr", [
    ("fp64", 1, 0, 2.0, 1.0), ("fp64", 3, 2, 10.0, 5.0),   # wider cells: sub-cell codes of nine bits leave room for the index
    ("split", 2, 3, 2.0, 1.0), ("split", 0, 2, 2.0, 1.0)])
def test_ordered_cells_equal_the_sorted_build(ks, precision, sub, spg, dt, thr):
    # Around the crowd size (256) and the part size (1024) of the ordering, with enough pairs to switch it on.
    st, sz, al = crowds(ks, [255, 256, 257, 300, 1023, 1024, 1025, 1300, 2047, 2049, 3072, 5000, 9000, 12000, 16000, 20000],
                        270_000)
    runs = []
    for form in (2, 0):
        with ks.Engine(0) as eng:
            eng.set_precision(ks.PRECISION_SPLIT if precision == "split" else ks.PRECISION_FP64)
            eng.set_tuning("sort_fused", form)
            eng.set_tuning("subcell_bits", sub)
            runs.append(run_engine(eng, st, sz, al, 9, dt=dt, thr=thr, spg=spg, chunks=[2, 3, 4]))
            assert eng.timing()["sort_cells_fused"] == form
    assert runs[0][3]["candidate_pairs"].max() > 600 * len(st)   # the bound above which cells are ordered
    assert len(runs[0][2]) > 0
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    assert_same_conj(runs[0][2], runs[1][2])
    assert_same_stats(runs[0][3], runs[1][3])


def test_one_shot_screening_of_crowds_equals_the_sorted_build(ks):
    st, sz, al = crowds(ks, [257, 1025, 5000, 9000], 270_000)
    with ks.Engine(0) as eng:
        eng.set_screening(True, 1.0, 1.0, 0.01)
        after, alive = eng.propagate(st, al, ks.DEFAULT_EPOCH_JD, 0.0, 2.0, 1)
        got = []
        for form in (2, 0):
            eng.set_tuning("sort_fused", form)
            c, s = eng.screen(st, after, alive, sz, 0.0, 2.0)
            got.append((c.copy(), s))
    assert len(got[0][0]) > 0
    assert_same_conj(got[0][0], got[1][0])
    for f in got[0][1].dtype.names:
        assert got[0][1][f] == got[1][1][f], f
