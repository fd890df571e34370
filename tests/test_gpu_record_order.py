"""Order of a chunk's records, at the sizes where the one-launch ordering changes shape."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_conj
from test_zz_no_alloc import crossing_groups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_group", [1, 3, 16, 33, 49, 68, 97, 113])
def test_records_of_one_step_in_order(ks, oracle, per_group):
    """per_group^2 records, all within a second of each other and many at
    equal times; run twice, so that the second run knows how many to expect and
    orders them in one launch (up to 12 900 in a step), then with more records
    than it takes (130^2 = 16 900), left to the multi-block sort."""
    with ks.Engine(0) as eng:
        eng.set_steps_per_graph(1)
        eng.set_screening(True, 5.0, 1.0, 0.01)
        for g in (per_group, per_group, 130):
            st, _, al, sz = crossing_groups(g)
            eng.set_clock(ks.DEFAULT_EPOCH_JD, 0.0, 10.0)
            eng.set_population(st, sz, al)
            eng.run(1)
            got = eng.take_conjunctions()
            want = oracle.run(st, sz, al, steps=1)[2]
            assert len(got) > 0
            assert_same_conj(got, want)
