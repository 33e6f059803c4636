"""GPU parity of the init passes around the size from which a thread takes several columns.

Graphs whose column counts sit on that size and on the edges of the passes' tiles
beyond it, with only short columns and with one long one (the general layout).
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1 << 17) - 1, 1 << 17, (1 << 17) + 1, (1 << 17) + 511, (1 << 17) + 769])
@pytest.mark.parametrize("longest", [2, 4, 5, 9])
def test_columns_per_thread(n, longest):
    rng = np.random.default_rng(n + longest)
    nv = n // 2
    a = rng.integers(0, nv, n - nv)
    rows = np.stack([a, (a + 1 + rng.integers(0, nv - 1, n - nv)) % nv], axis=1)
    rows.sort(axis=1)
    cols = [r for r in rows.astype(np.int32)]
    for at in (0, len(cols) // 2, len(cols) - 1):
        cols[at] = np.sort(rng.choice(nv, size=longest, replace=False)).astype(np.int32)
    dims = np.concatenate([np.zeros(nv, np.int32), np.ones(n - nv, np.int32)])
    lens = np.concatenate([np.zeros(nv, np.int64), [len(c) for c in cols]])
    order = rng.permutation(nv)  # vertices and edges interleaved, every edge after its vertices
    key = np.concatenate([order.astype(np.float64), [order[c].max() + 0.5 for c in cols]])
    seq = np.argsort(key, kind="stable")
    at = np.empty(n, np.int64)
    at[seq] = np.arange(n)
    entries = [np.empty(0, np.int32)] * nv + [np.sort(at[c]).astype(np.int32) for c in cols]
    m = BoundaryMatrix(dims[seq], np.concatenate([[0], np.cumsum(lens[seq])]).astype(np.int64),
                       np.concatenate([entries[i] for i in seq]).astype(np.int32))
    ref = oracle.reduce(m)
    with Engine(0) as e:
        e.load_csc(m)
        e.reduce(Params())
        assert np.array_equal(e.pairs(), ref.pairs)
        assert np.array_equal(e.essentials(), ref.essential)
