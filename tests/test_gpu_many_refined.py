"""Steps whose refinement outweighs the rest: run in one stream once a step has shown it."""
import numpy as np
import pytest

from test_gpu_memory import configured, results, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spg,chunks", [(0, [1, 2, 9]), (4, [36, 4]), (3, [3, 35, 2])])
def test_many_refined_pairs_per_object(ks, spg, chunks):
    """A cloud of 3 000 fragments an orbit old within 60 km: some 50 refined
    pairs an object (the bound is 40). Streams, and state buffers in turn, change between chunks;
    the results are those of the separate sort kernels."""
    st, sz, al = ks.generate_population(11, 2000, 5000, 1, 5000.0)
    got = []
    for form in (2, 0):
        with configured(ks, spg) as eng:
            eng.set_screening(True, 60.0, 1.0, 0.001)
            eng.set_tuning("sort_fused", form)
            eng.set_population(st, sz, al)
            eng.prepare_run()
            for k in chunks if form == 2 else [sum(chunks)]:
                eng.run(k)
            got.append(results(eng))
    refined = got[1][3]["refined_pairs"] / len(st)
    assert refined.max() > 40.0
    assert len(got[1][2]) > 1000
    same(*got)


@pytest.mark.parametrize("spg,chunks", [(4, [36, 3]), (0, [2, 40])])
def test_refinement_launched_before_the_tile_kernel_has_drained(ks, spg, chunks):
    """Large populations with a few refined pairs for every hundred objects: from
    the second chunk on the refinement starts early, in graphs and without."""
    st, sz, al = ks.generate_population(12, 28340, 270_000, 200, 86400.0)
    got = []
    for form in (2, 0):
        with configured(ks, spg) as eng:
            eng.set_screening(True, 12.0, 1.0, 0.01)
            eng.set_tuning("sort_fused", form)
            eng.set_population(st, sz, al)
            for k in chunks if form == 2 else [sum(chunks)]:
                eng.run(k)
            got.append(results(eng))
    refined = got[1][3]["refined_pairs"] / len(st)
    assert 0.005 < refined.min() and refined.max() < 1.0 and len(got[1][2]) > 1000
    same(*got)
