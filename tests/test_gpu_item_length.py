"""Length of the tile kernel's work items in a small population one of whose
clouds holds most of its pairs: it follows those pairs, in the first step too."""
import pytest

from test_gpu_memory import configured, holds_second, results, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fragments,age", [(2000, 600.0), (6500, 60.0), (9500, 60.0), (16000, 600.0), (43000, 600.0)])
def test_crowded_cells_equal_the_separate_kernels(ks, fragments, age):
    """Clouds around the bounds of the rule (15, 40 and 100 million pairs inside crowded cells)."""
    pop = ks.generate_population(77, 20000, 20000 + fragments, 1, age)
    got = []
    for form in (2, 0):
        with configured(ks, 2) as eng:
            eng.set_tuning("sort_fused", form)
            eng.set_population(*pop)
            eng.run(3)
            got.append(results(eng))
    assert got[1][3]["candidate_pairs"].max() > fragments ** 2 // 20
    same(*got)


def test_a_fresh_cloud_gets_long_items(ks):
    """43 000 fragments of one collision among 63 000 objects: items of the two
    column blocks that this population's size asks for would be some 450 000, above
    the 262 144 the list first holds; it would grow, and find no memory."""
    with configured(ks, 4) as eng:
        eng.set_population(*ks.generate_population(77, 20000, 63000, 1, 600.0))
        eng.prepare_run()
        eng.set_buffer_limits(1 << 23, 1 << 18)
        eng.set_tuning("deny_alloc", 1)
        eng.run(1)
        assert holds_second(ks, eng)
