"""Essentials of matrices that are no chain complexes.

Whatever the pairs of such a matrix are, its essentials are the columns in none of
them.  A column that owns a row from the start may lose the mark of an owner there:
its lowest row is removed with the negative rows when that row is a death itself.
"""
import numpy as np
import pytest

from specseqplusplus_b200 import Engine, Params, SsppError
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


def layers(rng, most):
    """Random columns of up to 8 rows of the dimension below, 2 to 5 dimensions of up to `most` cells."""
    count = [int(rng.integers(1, most)) for _ in range(int(rng.integers(2, 6)))]
    wide = int(rng.integers(2, 9))
    dims, cols, begin = [], [], 0
    for d, n in enumerate(count):
        for _ in range(n):
            k = int(rng.integers(0, min(wide, count[d - 1]) + 1)) if d else 0
            cols.append(begin + rng.choice(count[d - 1], size=k, replace=False))
            dims.append(d)
        if d:
            begin += count[d - 1]
    return BoundaryMatrix.from_columns(dims, [sorted(map(int, c)) for c in cols])


def unpaired(m, pairs):
    return np.setdiff1d(np.arange(m.ncols), pairs.reshape(-1))


@pytest.mark.parametrize("most,seeds", [(6, 60), (60, 60), (600, 20), (40_000, 1)])
@pytest.mark.parametrize("schedule", [0, 2])
def test_essentials_are_the_columns_in_no_pair(most, seeds, schedule):
    taken = 0
    with Engine(0) as e:
        for seed in range(seeds):
            m = layers(np.random.default_rng(seed), most)
            e.load_csc(m)
            try:
                e.reduce(Params(schedule=schedule))
            except SsppError as ex:  # a column that is a birth and a death from the start
                assert ex.code == 1
                continue
            taken += 1
            pairs = e.pairs()
            assert (np.diff(pairs[:, 0]) > 0).all()
            assert np.array_equal(e.essentials(), unpaired(m, pairs)), seed
    assert taken or most == 40_000


def test_an_owner_without_its_lowest_row():
    # edge 2 = {0, 1} takes row 1; edge 3 = {0} row 0; triangle 4 = {2, 3} owns row 3, which is negative,
    # as row 2 is: nothing is left of it
    m = BoundaryMatrix.from_columns([0, 0, 1, 1, 2], [[], [], [0, 1], [0], [2, 3]])
    with Engine(0) as e:
        e.load_csc(m)
        try:
            e.reduce(Params())
        except SsppError as ex:
            assert ex.code == 1
        else:
            assert np.array_equal(e.essentials(), unpaired(m, e.pairs()))


def test_batch():
    ms = []
    with Engine(0) as e:
        for seed in range(60):
            m = layers(np.random.default_rng(seed), 50)
            e.load_csc(m)
            try:
                e.reduce(Params())
            except SsppError:
                continue
            ms.append((m, e.pairs()))
        assert len(ms) > 5
        e.load_batch([m for m, _ in ms])
        e.reduce(Params())
        for (m, alone), (pairs, ess) in zip(ms, e.batch_results(), strict=True):
            assert np.array_equal(pairs, alone)
            assert np.array_equal(ess, unpaired(m, pairs))
