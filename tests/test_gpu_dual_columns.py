"""GPU parity of the dualization where its per-column work changes shape.

Stars give vertices dual columns of chosen lengths (one lane sorts up to 8 entries,
a warp up to 32 in registers and 1024 in shared memory, one block the rest); the
column counts are odd and even, since a lane takes a column and its mirror image.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params, gen
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


def check(m, **params):
    ref = oracle.reduce(m)
    with Engine(0) as e:
        e.load_csc(m)
        for _ in range(2):
            e.reduce(Params(**params))
            assert np.array_equal(e.pairs(), ref.pairs)
            assert np.array_equal(e.essentials(), ref.essential)


def stars(degrees, shift, seed):
    """Hubs with the given numbers of leaves among shared leaves, in a random order of edges."""
    rng = np.random.default_rng(seed)
    nv = len(degrees) + max(degrees) + shift
    edges = [(h, len(degrees) + int(x)) for h, k in enumerate(degrees)
             for x in rng.choice(max(degrees) + shift, size=k, replace=False)]
    rng.shuffle(edges)
    return BoundaryMatrix.from_columns([0] * nv + [1] * len(edges), [[]] * nv + [sorted(map(int, x)) for x in edges])


@pytest.mark.parametrize("dualize", [1, 2])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("degrees", [[1], [2, 3, 4], [4, 5, 7, 8, 9], [31, 32, 33], [1, 63, 64, 65, 2], [1023, 1024, 1025, 3],
                                     [5000, 8191, 8193]])
def test_lengths_of_dual_columns(degrees, shift, dualize):
    check(stars(degrees, shift, sum(degrees)), dualize=dualize)


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 63, 64, 65, 511, 512, 513])
@pytest.mark.parametrize("dualize", [1, 2])
def test_counts_of_columns(n, dualize):
    # one edge, the rest vertices, then the edge in the middle of them
    for at in (n - 1, n // 2):
        cols = [[]] * n
        if at >= 2:
            cols = cols[:at] + [[0, at - 1]] + cols[at + 1:]
        check(BoundaryMatrix.from_columns([1 if c else 0 for c in cols], cols), dualize=dualize)


@pytest.mark.parametrize("dualize", [1, 2])
@pytest.mark.parametrize("schedule", [1, 2])
def test_cofaces_of_every_dimension(dualize, schedule):
    rng = np.random.default_rng(3)
    m = gen.rips_from_points(rng.random((70, 3)).astype(np.float32), 0.55, 3)
    check(m, dualize=dualize, schedule=schedule)


@pytest.mark.parametrize("dualize", [1, 2])
def test_dropped_columns(dualize):
    rng = np.random.default_rng(4)
    m = gen.rips_from_points(rng.random((120, 2)).astype(np.float32), 0.3, 2)
    out = []
    with Engine(0) as e:
        e.load_csc(m)
        for d in (0, dualize):
            e.reduce(Params(model=2, dualize=d))
            out.append((e.pairs(), e.essentials()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
