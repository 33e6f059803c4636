"""Batches whose many small arrays are staged together.

Up to 1 MB they go through the buffer of small copies, beyond it through the
large one; a load's staging waits for the copies of the load before it.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params, gen
from specseqplusplus_b200.gen import BoundaryMatrix
from test_gpu_small_copies import ring

pytestmark = pytest.mark.gpu


def check(e, mats):
    for m, (pairs, ess) in zip(mats, e.batch_results(), strict=True):
        want = oracle.reduce(m)
        assert np.array_equal(pairs, want.pairs)
        assert np.array_equal(ess, want.essential)


# 12 bytes a vertex and 20 an edge, 160 for the starts: 3,460 edges of the last complex bring the
# batch to 2^20 bytes exactly
@pytest.mark.parametrize("edges", [0, 17, 3460, 3461])
def test_sizes_around_the_limit(edges):
    mats = [ring(100 + i, 10 + i) for i in range(7)] + [ring(40_000, 22_036), ring(4002, edges)]
    with Engine(0) as e:
        for _ in range(2):
            e.load_batch(mats)
            e.reduce(Params())
            check(e, mats)


def test_loads_one_after_another():
    empty = BoundaryMatrix.from_columns([], [])
    a = [ring(20 + i, 5 + i) for i in range(30)] + [empty] * 3
    b = [empty] + [gen.rips(60, 3, s, 0.4, 3) for s in range(12)]
    one = [ring(500, 400)]
    clouds = [("rips", gen.points(30 + i, 2, i), 0.3, 2) for i in range(20)]
    with Engine(0) as e:
        for _ in range(3):
            for earlier in (a, b, one):
                for m in (a, b):
                    e.load_batch(earlier)
                    e.load_csc(one[0])
                    e.load_batch(m)
                    e.reduce(Params())
                    check(e, m)
            e.load_batch(a)
            e.load_built_batch(clouds)
            e.reduce(Params())
            check(e, [gen.rips_from_points(c[1], c[2], c[3]) for c in clouds])
