"""The autotuner's candidates are different runs.

Block size and growth take effect in schedule 2 alone, and the warp tier holds at
most 64 ints a column, so settings are told apart by what is left of them.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("autotune,schedule,radius", [(1, 0, 0.01), (2, 0, 0.01), (1, 2, 0.0003)])
def test_candidates_differ_in_what_takes_effect(autotune, schedule, radius):
    # graphs with guided clearing, mostly edges or mostly vertices: classes that no other test
    # measures, so no candidate is left out for what it took there
    m = gen.rips(1500, 1, 4, radius, 1)
    want = oracle.reduce(m)
    seen = {}
    with Engine(0) as e:
        for _ in range(9):
            e.load_csc(m)
            e.reduce(Params(autotune=autotune, schedule=schedule, model=1, max_iteration=3))
            p = e.params()
            c = e.stats()["tuned_candidate"]
            own = (min(max(p.level1_capacity, 32), 64), p.level2_capacity, p.heavy_threads, p.dualize)
            assert seen.setdefault(c, own) == own
            assert np.array_equal(e.pairs(), want.pairs)
            assert np.array_equal(e.essentials(), want.essential)
    assert len(set(seen.values())) == len(seen) >= 4
