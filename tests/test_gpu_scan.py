"""GPU parity at the sizes where the one-pass scans change shape.

Column counts around one tile (4,096), around 32 tiles (the look-back's width) and
beyond, with matrices whose offsets, active lists, pairs and essentials all pass
through a scan of that many items.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


def random_edges(n, seed):
    """n cells: vertices and edges between earlier vertices, in a random order of dimensions."""
    rng = np.random.default_rng(seed)
    dims = (rng.random(n) < 0.6).astype(np.int32)
    dims[:2] = 0
    nv = np.cumsum(dims == 0) - (dims == 0)  # vertices before each cell
    vert = np.flatnonzero(dims == 0).astype(np.int32)
    e = np.flatnonzero(dims == 1)
    a = (rng.random(e.size) * nv[e]).astype(np.int64)
    b = (a + 1 + (rng.random(e.size) * (nv[e] - 1)).astype(np.int64)) % nv[e]
    rows = np.stack([vert[np.minimum(a, b)], vert[np.maximum(a, b)]], axis=1)
    col_ptr = np.concatenate([[0], np.cumsum(2 * (dims == 1))]).astype(np.int64)
    return BoundaryMatrix(dims, col_ptr, rows.reshape(-1).astype(np.int32))


@pytest.mark.parametrize("n", [2, 31, 4095, 4096, 4097, 8192, 8193, 32 * 4096, 33 * 4096, 33 * 4096 + 1, 65 * 4096 + 17])
@pytest.mark.parametrize("dualize", [0, 1])
def test_column_counts_around_the_tiles(n, dualize):
    if dualize and n > 9000:
        pytest.skip("the dual of a random graph has long vertex columns")
    m = random_edges(n, n)
    ref = oracle.reduce(m)
    with Engine(0) as e:
        for _ in range(2):
            e.load_csc(m)
            e.reduce(Params(dualize=dualize))
            assert np.array_equal(e.pairs(), ref.pairs)
            assert np.array_equal(e.essentials(), ref.essential)


def test_dimensions_without_columns():
    # dimensions 0, 2, 3 and 5: cells without a boundary, and one 3-cell over a 2-cell
    dims = [0, 5, 2, 2, 3, 5, 0]
    m = BoundaryMatrix.from_columns(dims, [[], [], [], [], [2, 3], [], []])
    ref = oracle.reduce(m)
    with Engine(0) as e:
        e.load_csc(m)
        for schedule in (1, 2):
            e.reduce(Params(schedule=schedule))
            assert np.array_equal(e.pairs(), ref.pairs)
            assert np.array_equal(e.essentials(), ref.essential)
