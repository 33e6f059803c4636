"""What the allocation-free call does with the caller's buffers.

They are int64 arrays: a pool that hands out slices of its own memory may start
them on any 8-byte boundary.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import gen
from specseqplusplus_b200.engine import reduce_noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("npts", [6, 60, 700])  # the one-block kernel, one tile of the pairs' scan, several
def test_pairs_on_any_eight_byte_boundary(npts, shift):
    torch = pytest.importorskip("torch")
    m = gen.rips(npts, 3, 21, gen.rips_radius_for_degree(npts, 3, min(8.0, npts / 3)), 3)
    want = oracle.reduce(m).pairs
    dims, col_ptr, rows = (torch.from_numpy(x).cuda() for x in (m.dims, m.col_ptr, m.rows))
    pool = torch.full((2 * m.ncols + 8,), -7, dtype=torch.int64, device="cuda")
    assert pool.data_ptr() % 16 == 0
    pairs, npairs = pool[4 + shift:], pool[shift:shift + 1]
    reduce_noalloc(m.ncols, m.nnz, dims.data_ptr(), col_ptr.data_ptr(), rows.data_ptr(), pairs.data_ptr(),
                   npairs.data_ptr(), torch.cuda.current_stream().cuda_stream)
    k = int(npairs.item())
    got = pool.cpu().numpy()
    assert k == len(want)
    assert np.array_equal(got[4 + shift:4 + shift + 2 * k].reshape(-1, 2), want)
    # and nothing else of the pool
    rest = np.delete(got, np.r_[shift, 4 + shift:4 + shift + 2 * k])
    assert (rest == -7).all()
