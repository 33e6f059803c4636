"""GPU parity where a scan's tile looks back over more than one window.

A tile reads the states of the 256 before it at a time; scans of numbers, of classes
and of bytes beyond 2^18 items have tiles of 4,096.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu

WINDOW = 256 * 4096


def path(n, seed, extra=0):
    """n cells in a random order of dimensions: vertices, and edges between neighbours of a path; one column
    with `extra` more rows, so that not every column is short and the slots' offsets are scanned too."""
    rng = np.random.default_rng(seed)
    dims = (rng.random(n) < 0.6).astype(np.int32)
    dims[:2] = 0
    vert = np.flatnonzero(dims == 0).astype(np.int32)
    e = np.flatnonzero(dims == 1)
    nv = np.cumsum(dims == 0)[e]  # vertices before each edge
    a = (rng.random(e.size) * (nv - 1)).astype(np.int64)
    rows = np.stack([vert[a], vert[a + 1]], axis=1).reshape(-1)
    lens = 2 * (dims == 1).astype(np.int64)
    if extra:
        lens[e[-1]] = 2 + extra
        rows = np.concatenate([rows[:-2], vert[:2 + extra]])
    return BoundaryMatrix(dims, np.concatenate([[0], np.cumsum(lens)]), rows.astype(np.int32))


@pytest.mark.parametrize("n", [WINDOW - 1, WINDOW, WINDOW + 1, 2 * WINDOW + 4097])
@pytest.mark.parametrize("extra,dualize", [(0, 0), (0, 2), (4, 0)])
def test_column_counts_around_the_windows(n, extra, dualize):
    m = path(n, n, extra)
    ref = oracle.reduce(m)
    with Engine(0) as e:
        for _ in range(2):
            e.load_csc(m)
            e.reduce(Params(dualize=dualize))
            assert np.array_equal(e.pairs(), ref.pairs)
            assert np.array_equal(e.essentials(), ref.essential)
