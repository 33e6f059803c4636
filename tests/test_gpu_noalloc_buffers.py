"""What the allocation-free call does with the caller's buffers.

They are int64 arrays: a pool that hands out slices of its own memory may start
them on any 8-byte boundary.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import SsppError, gen
from specseqplusplus_b200.engine import reduce_noalloc
from specseqplusplus_b200.gen import BoundaryMatrix
from test_gpu_noalloc_scratch import twist_pairs
from test_zz_no_alloc import _noalloc_pairs

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


@pytest.mark.parametrize("ncols", [1, 2, 51, 223, 224, 225, 226])  # up to 224: the one-block kernel alone
def test_columns_around_the_smallest_of_the_passes(ncols):
    torch = pytest.importorskip("torch")
    m = gen.rips(64, 3, 5, 0.4, 3)
    m = BoundaryMatrix(m.dims[:ncols], m.col_ptr[:ncols + 1], m.rows[:m.col_ptr[ncols]])  # a subcomplex
    assert m.ncols == ncols
    assert np.array_equal(_noalloc_pairs(m, torch), oracle.reduce(m).pairs)


@pytest.mark.parametrize("seed", range(20))
def test_larger_matrices_that_are_not_chain_complexes(seed):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(seed)
    layer = [int(rng.integers(120, 400)) for _ in range(int(rng.integers(2, 5)))]
    dims, cols, begin = [], [], 0
    for d, n in enumerate(layer):
        for _ in range(n):
            k = 0 if d == 0 else int(rng.integers(0, 7))
            cols.append(begin + rng.choice(layer[d - 1], size=k, replace=False) if k else [])
            dims.append(d)
        if d:
            begin += layer[d - 1]
    m = BoundaryMatrix.from_columns(dims, cols)
    assert m.ncols > 224 and np.array_equal(_noalloc_pairs(m, torch), twist_pairs(m))


def _long_columns(k):
    """Edges {r - 1, r} own the rows 1..4095; each of k columns {0..4095} after them takes 2,048 of their
    additions and comes out zero, 4,196,352 ints of fill-in with new room for every one."""
    nv = 4096
    dims = np.concatenate([np.zeros(nv, np.int32), np.ones(nv - 1 + k, np.int32)])
    lens = np.concatenate([np.zeros(nv), np.full(nv - 1, 2), np.full(k, nv)]).astype(np.int64)
    rows = np.concatenate([np.stack([np.arange(nv - 1), np.arange(1, nv)], 1).reshape(-1), np.tile(np.arange(nv), k)])
    m = BoundaryMatrix(dims, np.concatenate([[0], np.cumsum(lens)]), rows.astype(np.int32))
    return m, np.stack([np.arange(1, nv), nv + np.arange(nv - 1)], 1)


def _short_chains(k, rows):
    """Edges {r - 1, r} own the rows 1..rows; k columns {0, rows} after them take one addition after
    another down to row 0: four ints each, within what the parallel account holds on chip."""
    dims = np.concatenate([np.zeros(rows + 1, np.int32), np.ones(rows + k, np.int32)])
    col_ptr = np.concatenate([np.zeros(rows + 1, np.int64), 2 * np.arange(rows + k + 1, dtype=np.int64)])
    r = np.concatenate([np.stack([np.arange(rows), np.arange(1, rows + 1)], 1).reshape(-1), np.tile([0, rows], k)])
    return BoundaryMatrix(dims, col_ptr, r.astype(np.int32)), np.stack([np.arange(1, rows + 1), 2 * rows + 1 - np.arange(rows, 0, -1)], 1)


def fill_in(m):
    """(ints that the additions of a twist reduction in column order read, room for them in the array)"""
    cols = [set(map(int, m.column(j))) for j in range(m.ncols)]
    owner, total = {}, 0
    for d in range(int(m.dims.max()), 0, -1):
        for j in np.flatnonzero(m.dims == d):
            while cols[j] and max(cols[j]) in owner:
                add = cols[owner[max(cols[j])]]
                total += len(cols[j]) + len(add)
                cols[j] = cols[j] ^ add
            if cols[j]:
                owner[max(cols[j])] = int(j)
                cols[max(cols[j])] = set()
    return total, (16 << 20) - 16 - 3 * m.ncols - m.nnz


@pytest.mark.parametrize("k,fits", [(3, True), (4, False), (250, False)])
def test_fill_in_of_long_columns_is_judged_alike_every_time(k, fits):
    torch = pytest.importorskip("torch")
    m, want = _long_columns(k)
    # 2,048 additions of 4096, 4094, ... 2 entries, and two more each
    room = (16 << 20) - 16 - 3 * m.ncols - m.nnz
    assert (k * (2048 * 2049 + 2 * 2048) <= room) == fits
    for _ in range(4):
        if fits:
            assert np.array_equal(_noalloc_pairs(m, torch), want)
            continue
        with pytest.raises(SsppError) as ei:
            _noalloc_pairs(m, torch)
        assert ei.value.code == 2 and "scratch" in str(ei.value)


@pytest.mark.parametrize("over", [-1, 1])
def test_fill_in_of_short_columns_right_at_the_limit(over):
    torch = pytest.importorskip("torch")
    # four ints an addition: the number of chains of 500 decides on which side of the room they end
    rows = 500
    small, _ = _short_chains(3, rows)
    per = fill_in(small)[0] // 3
    assert per == 4 * rows
    k = 1
    while k * per <= (16 << 20) - 16 - 3 * (2 * rows + 1 + k) - 2 * (rows + k):
        k += 1  # the first number of chains that does not fit
    m, want = _short_chains(k - 1 if over < 0 else k, rows)
    for _ in range(3):
        if over < 0:
            assert np.array_equal(_noalloc_pairs(m, torch), want)
        else:
            with pytest.raises(SsppError) as ei:
                _noalloc_pairs(m, torch)
            assert ei.value.code == 2 and "scratch" in str(ei.value)


def test_refused_fill_in_writes_nothing():
    torch = pytest.importorskip("torch")
    # 6,000 columns of 50 random rows out of 12,000: reduced they are thousands of rows long,
    # some 27 M ints, more than either way through the array has room for
    nv, ne = 12_000, 6_000
    rng = np.random.default_rng(1)
    rows = np.sort(np.stack([rng.choice(nv, 50, replace=False) for _ in range(ne)]), axis=1)
    dims = np.concatenate([np.zeros(nv, np.int32), np.ones(ne, np.int32)])
    col_ptr = np.concatenate([np.zeros(nv, np.int64), 50 * np.arange(ne + 1, dtype=np.int64)])
    d = [torch.from_numpy(x).cuda() for x in (dims, col_ptr, rows.reshape(-1).astype(np.int32))]
    out = torch.full((2 * (nv + ne) + 1,), -7, dtype=torch.int64, device="cuda")
    for _ in range(2):
        with pytest.raises(SsppError) as ei:
            reduce_noalloc(nv + ne, 50 * ne, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out[1:].data_ptr(),
                           out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert ei.value.code == 2 and "scratch" in str(ei.value)
        assert bool((out == -7).all())
    m = gen.lowerstar(10, 1.0, 9)
    assert np.array_equal(_noalloc_pairs(m, torch), oracle.reduce(m).pairs)
