"""More pairs than half the columns.

A matrix that is no chain complex may pair a column twice, as a birth and as a
death.  Each unit here has a vertex v, an edge b = {v}, an edge x without a
boundary and the triangles {x} and {b, x}: with the columns kept whole
(representatives) its pairs are (v, b), (x, {x}) and (b, {b, x}), three of five
columns.
"""
import numpy as np
import pytest

from specseqplusplus_b200 import Engine, Params
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


def units(k):
    """(matrix, pairs, essentials): k vertices, then b x of each unit, then its triangles"""
    i = np.arange(k)
    b, x = k + 2 * i, k + 2 * i + 1
    t = 3 * k + 2 * i  # {x}; t + 1 = {b, x}
    dims = np.concatenate([np.zeros(k), np.ones(2 * k), np.full(2 * k, 2)]).astype(np.int32)
    lens = np.concatenate([np.zeros(k), np.tile([1, 0], k), np.tile([1, 2], k)]).astype(np.int64)
    col_ptr = np.concatenate([[0], np.cumsum(lens)])
    rows = np.concatenate([i, np.stack([x, b, x], axis=1).reshape(-1)]).astype(np.int32)
    pairs = np.concatenate([np.stack([i, b], 1), np.stack([x, t], 1), np.stack([b, t + 1], 1)])
    return BoundaryMatrix(dims, col_ptr, rows), pairs[np.argsort(pairs[:, 0])], np.zeros(0, np.int64)


@pytest.mark.parametrize("k", [1, 100, 10922, 10923, 13000, 13107, 13108, 40000])  # around 2^15 pairs and 2^16 columns
def test_pairs_of_columns_that_are_in_two(k):
    m, want, ess = units(k)
    with Engine(0) as e:
        for _ in range(2):
            e.load_csc(m)
            e.reduce(Params(representatives=1))
            assert e.num_pairs() == 3 * k
            assert np.array_equal(e.pairs(), want)
            assert np.array_equal(e.essentials(), ess)


def test_batch_of_such_matrices():
    sizes = [1, 2000, 70, 900, 5]
    cases = [units(k) for k in sizes]
    with Engine(0) as e:
        for _ in range(2):
            e.load_batch([m for m, _, _ in cases])
            e.reduce(Params(representatives=1))
            for (pairs, ess), (_, want, none) in zip(e.batch_results(), cases):
                assert np.array_equal(pairs, want)
                assert np.array_equal(ess, none)
