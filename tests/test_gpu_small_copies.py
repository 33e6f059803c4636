"""GPU parity around the sizes up to which one kernel moves inputs and results.

Inputs of at most 1 MB are fetched by a kernel from pinned memory that the load
fills and does not wait for; results of at most 65,536 columns are written to pinned
memory by the reduction itself.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


def ring(nv, ne):
    """nv vertices and ne edges between neighbours of a ring, in order."""
    dims = np.concatenate([np.zeros(nv, np.int32), np.ones(ne, np.int32)])
    col_ptr = np.concatenate([np.zeros(nv, np.int64), 2 * np.arange(ne + 1, dtype=np.int64)])
    rows = np.stack([np.arange(ne) % nv, (np.arange(ne) + 1) % nv], axis=1)
    rows.sort(axis=1)
    return BoundaryMatrix(dims, col_ptr, rows.reshape(-1).astype(np.int32))


def results(e):
    return e.pairs(), e.essentials()


def same(got, m):
    ref = oracle.reduce(m)
    assert np.array_equal(got[0], ref.pairs) and np.array_equal(got[1], ref.essential)


# 12 bytes a vertex and 20 an edge, 8 more: 2^20 bytes are 65,536 columns short of 32,767.5 edges
@pytest.mark.parametrize("nv,ne", [(2, 1), (1, 0), (32768, 32767), (32768, 32768), (32769, 32768), (20000, 40428),
                                   (20000, 40429), (20001, 40428), (60000, 5535), (60000, 5536), (60000, 5537)])
def test_sizes_around_the_limits(nv, ne):
    m = ring(nv, ne)
    with Engine(0) as e:
        e.load_csc(m)
        e.reduce(Params())
        same(results(e), m)


def test_loads_one_after_another_and_other_streams():
    torch = pytest.importorskip("torch")
    ms = [ring(500, 400), ring(70, 900), ring(60000, 5000), ring(3, 2)]
    side = torch.cuda.Stream()
    with Engine(0) as e:
        for stream in (0, side.cuda_stream, 0):
            for m in ms:  # the later load's staging waits for the earlier fetch
                e.load_csc(ms[0])
                e.load_csc(m)
                e.reduce(Params(), stream)
                same(results(e), m)
            for m in ms[:2]:
                e.load_csc(m)
            for _ in range(2):  # the input stays for another reduction
                e.reduce(Params(), stream)
                same(results(e), ms[1])


@pytest.mark.parametrize("nv,ne", [(500, 400), (60000, 9000)])
def test_result_buffers(nv, ne):
    torch = pytest.importorskip("torch")
    m = ring(nv, ne)
    ref = oracle.reduce(m)
    pinned = [torch.full((2 * m.ncols,), -1, dtype=torch.int64).pin_memory().numpy() for _ in range(2)]
    plain = [np.full(2 * m.ncols, -1, np.int64) for _ in range(2)]
    odd = [np.frombuffer(bytearray(16 * m.ncols + 4), np.uint8)[4:].view(np.int64) for _ in range(2)]
    with Engine(0) as e:
        e.load_csc(m)
        e.reduce(Params())
        for a, b in (pinned, plain, odd):
            assert np.array_equal(e.pairs(a), ref.pairs) and np.array_equal(e.essentials(b), ref.essential)
        assert (plain[0][ref.pairs.size:] == -1).all() and (pinned[1][ref.essential.size:] == -1).all()
