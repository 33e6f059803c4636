"""GPU parity of the reduction's rounds of additions against the oracle.

A round takes a column's top rows, one per thread of the group, adds every
owner that is an earlier column, sorts what the addends leave in runs of 64
entries and merges it into the rest of the column.  The matrices here are free
of geometry: the rows are cells without a boundary, so every column of the next
dimension may hold any set of rows, and column lengths, addend lengths and the
number of additions are chosen to sit on the edges of those sizes.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


def matrix(nrows, columns):
    """nrows cells without a boundary, then one cell of the next dimension per column."""
    dims = np.concatenate([np.ones(nrows, np.int32), np.full(len(columns), 2, np.int32)])
    cols = [np.unique(np.asarray(c, dtype=np.int32)) for c in columns]
    lens = np.concatenate([np.zeros(nrows, np.int64), [len(c) for c in cols]])
    return BoundaryMatrix(dims, np.concatenate([[0], np.cumsum(lens)]).astype(np.int64),
                          np.concatenate(cols).astype(np.int32))


def check(m, p):
    ref = oracle.reduce(m)
    with Engine(0) as e:
        e.load_csc(m)
        e.reduce(p)
        assert np.array_equal(e.pairs(), ref.pairs)
        assert np.array_equal(e.essentials(), ref.essential)


LENGTHS = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1025, 3000]


@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("l1,l2", [(32, 96), (32, 8192), (1000, 8000)])
def test_long_columns_over_short_owners(threads, l1, l2):
    # owners {r, two rows below} of every row but some, then columns whose lengths are the group's sizes and one off
    rng = np.random.default_rng(7)
    n = 4000
    cols = []
    for r in range(8, n):
        if r % 7:
            cols.append([r] + list(rng.integers(max(0, r - 60), r, size=rng.integers(0, 5))))
    rng.shuffle(cols)
    for length in LENGTHS:
        cols.append(rng.choice(n, size=length, replace=False))
        cols.append(np.arange(n - length, n))
    check(matrix(n, cols), Params(level1_capacity=l1, level2_capacity=l2, heavy_threads=threads))


@pytest.mark.parametrize("length", [1, 2, 4, 5, 31, 32, 33, 64])
@pytest.mark.parametrize("l1,l2", [(32, 64), (64, 8192)])
def test_owners_of_every_addend_length(length, l1, l2):
    # published owners (each row's column comes second, so that no owner is an apparent pair) of one length
    rng = np.random.default_rng(length)
    n = 700
    cols = []
    for r in range(length, n):
        low = rng.choice(r, size=length - 1, replace=False)
        cols.append(np.append(low, r))
    cols += [rng.choice(n, size=k, replace=False) for k in (3, 17, 32, 33, 100, 256, 300, 513, 650)]
    check(matrix(n, cols), Params(level1_capacity=l1, level2_capacity=l2, ss_block_size=200, growth=1.0))


@pytest.mark.parametrize("seed", range(6))
def test_random_matrices(seed):
    # dense fill-in, duplicates that cancel, empty results; capacities that force both tiers and arena columns
    rng = np.random.default_rng(100 + seed)
    n = int(rng.integers(20, 600))
    cols = [rng.choice(n, size=int(rng.integers(1, min(n, 40))), replace=False) for _ in range(2 * n)]
    for l1, l2 in ((32, 32), (32, 128), (256, 4096)):
        check(matrix(n, cols), Params(level1_capacity=l1, level2_capacity=l2, ss_block_size=1 + 97 * seed, growth=1.2))
