"""GPU parity of the allocation-free call's two ways through the scratch array.

The engine's passes run in it while their arrays fit; larger inputs, and runs
that do not end cleanly, go to the one-block kernel.  Both must give the twist
reduction's pairs for every well-formed matrix, also when the boundary of a
boundary is not zero.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import gen
from specseqplusplus_b200.gen import BoundaryMatrix
from test_zz_no_alloc import _noalloc_pairs

pytestmark = pytest.mark.gpu


def twist_pairs(m):
    """Dimensions from high to low, columns in order, cleared when their row is claimed."""
    cols = [set(map(int, m.column(j))) for j in range(m.ncols)]
    owner = {}
    for d in range(int(m.dims.max()), 0, -1):
        for j in np.flatnonzero(m.dims == d):
            while cols[j] and max(cols[j]) in owner:
                cols[j] ^= cols[owner[max(cols[j])]]
            if cols[j]:
                low = max(cols[j])
                owner[low] = int(j)
                cols[low] = set()
    return np.array(sorted(owner.items()), dtype=np.int64).reshape(-1, 2)


@pytest.mark.parametrize("seed", range(20))
def test_matrices_that_are_not_chain_complexes(seed):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(seed)
    layer = [int(rng.integers(1, 40)) for _ in range(int(rng.integers(2, 5)))]
    dims, cols, begin = [], [], 0
    for d, n in enumerate(layer):
        for _ in range(n):
            k = 0 if d == 0 else int(rng.integers(0, min(6, layer[d - 1]) + 1))
            cols.append(begin + rng.choice(layer[d - 1], size=k, replace=False) if k else [])
            dims.append(d)
        if d:
            begin += layer[d - 1]
    m = BoundaryMatrix.from_columns(dims, cols)
    assert np.array_equal(_noalloc_pairs(m, torch), twist_pairs(m))


@pytest.mark.parametrize("grid", [2, 3, 12, 20])
def test_grids_in_the_scratch_array(grid):
    torch = pytest.importorskip("torch")
    m = gen.lowerstar(grid, 1.5, 3)
    assert np.array_equal(_noalloc_pairs(m, torch), oracle.reduce(m).pairs)


@pytest.mark.parametrize("ncols", [1, 2, 255, 256, 257])
def test_columns_without_a_boundary(ncols):
    torch = pytest.importorskip("torch")
    m = BoundaryMatrix.from_columns([0] * ncols, [[]] * ncols)
    assert len(_noalloc_pairs(m, torch)) == 0


def test_larger_than_the_scratch_passes_take():
    # 900,000 columns: 67 bytes each and their slots exceed the array, so the one-block kernel runs
    torch = pytest.importorskip("torch")
    n = 450_000
    dims = np.concatenate([np.zeros(n, np.int32), np.ones(n, np.int32)])
    col_ptr = np.concatenate([np.zeros(n, np.int64), 2 * np.arange(n + 1, dtype=np.int64)])
    rows = np.stack([np.arange(n), (np.arange(n) + 1) % n], axis=1)
    rows.sort(axis=1)
    m = BoundaryMatrix(dims, col_ptr, rows.reshape(-1).astype(np.int32))
    got = _noalloc_pairs(m, torch)
    assert np.array_equal(got, oracle.reduce(m).pairs)
