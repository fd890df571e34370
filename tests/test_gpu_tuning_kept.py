"""What the autotuner leaves in place beside the configuration it chose."""
import numpy as np
import pytest

from test_gpu_memory import configured, holds_second

pytestmark = pytest.mark.gpu


def test_item_length_by_the_population_outlives_a_tuning_of_another(ks):
    """A tuning that keeps its starting configuration (here: one that a barrier
    limit of no polls ends) leaves the length of a work item to the population.
    The length that 2 000 objects give (2 column blocks) would make 480 000 items
    of the second population, above the 262 144 the list first holds (126 000 at
    its own length, 8): the list would grow, and find no memory."""
    with configured(ks, 4, 20.0) as eng:
        eng.set_population(*ks.generate_population(3, 2000))
        eng.set_tuning("sort_fused", 1)
        eng.set_tuning("lookback_polls", 0)
        for _ in range(10):   # whether a barrier is found incomplete is a race
            try:
                eng.autotune(1)
            except ks.KsError:
                break
            eng.set_tuning("item_col_blocks", 0)
        else:
            raise AssertionError("no barrier wait ran out in 10 tunings")
        eng.set_tuning("lookback_polls", 1 << 22)
        eng.set_tuning("sort_fused", 2)
        eng.set_population(*ks.generate_population(17, 28340, 400000, 60, 3600.0))
        eng.prepare_run()
        eng.set_buffer_limits(1 << 21, 1 << 18)
        eng.set_tuning("deny_alloc", 1)
        eng.run(4)
        assert holds_second(ks, eng)


@pytest.mark.parametrize("block", [32, 96])
def test_tuning_without_screening_times_the_steps_a_run_takes(ks, oracle, block):
    """Without screening a run carries many steps a launch: the graph length says
    nothing there and is not tried; the threads per block are."""
    st, sz, al = ks.generate_population(8, 3001)
    with configured(ks, 0) as eng:
        eng.set_screening(False)
        eng.set_tuning("prop_block", block)
        eng.set_population(st, sz, al)
        choice = eng.autotune(130)
        # The start and the block sizes; a starting size among them is tried again where another has beaten it.
        assert choice["trials"] - 1 in ((3,) if block == 32 else (2, 3))
        assert choice["steps_per_graph"] == 0
        assert eng.clock() == (0.0, 0) and len(eng.take_step_stats()) == 0
        eng.set_tuning("prop_block", block)
        eng.run(140)
        fs, fa = eng.get_population()
    want = oracle.run(st, sz, al, steps=140, screen=False)
    assert np.array_equal(fs, want[0]) and np.array_equal(fa, want[1])


def test_packed_keys_return_after_a_tuning_trial_too_wide_for_them(ks):
    """Sub-cell bits tried by the tuner widen the keys past the room for the
    object index; the configuration it leaves has them packed again and so
    builds its cells by counting."""
    st, sz, al = ks.generate_population(31, 5000)   # 15 bits an axis at these cells: no room for a second sub-cell bit
    with configured(ks, 8, 0.1) as eng:
        eng.set_screening(True, 2.0, 1.0, 0.01)
        eng.set_population(st, sz, al)
        for sub in (2, 1):
            eng.set_tuning("subcell_bits", sub)
            eng.run(1)
            assert (eng.timing()["sort_cells_fused"] == 2) == (sub == 1)
        choice = eng.autotune(1)
        assert choice["subcell_bits"] <= 1
        eng.set_tuning("pair_variant", 2)
        eng.run(1)
        assert eng.timing()["sort_cells_fused"] == 2
