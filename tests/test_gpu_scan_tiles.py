"""GPU parity at the column counts where the scans change the size of their tiles."""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096, 4097, 5120, 5121, 32 * 1024 + 1, (1 << 18) - 1, 1 << 18, (1 << 18) + 1])
@pytest.mark.parametrize("longest,dualize", [(2, 0), (2, 2), (5, 0)])  # 5: the slots' offsets are scanned too
def test_tile_sizes(n, longest, dualize):
    # a path, closed to a ring at the end, and vertices of their own; one longer column
    ne = 2 * n // 5
    nv = n - ne
    cols = np.stack([np.arange(ne) % nv, (np.arange(ne) + 1) % nv], axis=1)
    cols.sort(axis=1)
    lens = np.concatenate([np.zeros(nv, np.int64), np.full(ne, 2, np.int64)])
    rows = cols.reshape(-1)
    if longest > 2:
        lens[-1] = longest
        rows = np.concatenate([rows[:-2], np.arange(nv - longest, nv)])
    dims = np.concatenate([np.zeros(nv, np.int32), np.ones(ne, np.int32)])
    m = BoundaryMatrix(dims, np.concatenate([[0], np.cumsum(lens)]).astype(np.int64), rows.astype(np.int32))
    ref = oracle.reduce(m)
    with Engine(0) as e:
        e.load_csc(m)
        for _ in range(2):
            e.reduce(Params(dualize=dualize))
            assert np.array_equal(e.pairs(), ref.pairs)
            assert np.array_equal(e.essentials(), ref.essential)
