"""A matrix that the compression pass refuses while its blocks are still starting.

Columns that are apparent deaths and births at once exist only without the chain
property; the pass that meets one sets the error word, which its other blocks look
at when they start.  The call must end as a malformed input and leave the context
as it was.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params, SsppError, gen
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 150_000])
@pytest.mark.parametrize("model", [0, 1])
def test_columns_that_are_births_and_deaths(n, model):
    # edge i = {vertex i}, triangle i = {edge i}
    dims = np.repeat(np.arange(3, dtype=np.int32), n)
    col_ptr = np.concatenate([np.zeros(n, np.int64), np.arange(2 * n + 1, dtype=np.int64)])
    m = BoundaryMatrix(dims, col_ptr, np.arange(2 * n, dtype=np.int32))
    good = gen.lowerstar(12, 1.5, 3)
    want = oracle.reduce(good)
    p = Params(model=model, max_iteration=10)
    with Engine(0) as e:
        for _ in range(3):
            e.load_csc(m)
            with pytest.raises(SsppError) as ei:
                e.reduce(p)
            assert ei.value.code == 1 and "malformed" in str(ei.value)
            e.load_csc(good)
            e.reduce(p)
            assert np.array_equal(e.pairs(), want.pairs)
            assert np.array_equal(e.essentials(), want.essential)
