"""GPU parity of complexes built together with the host builder's, bit for bit.

A batch's consecutive point clouds are built as one block-diagonal graph: one
cell grid per cloud, one neighbour search, one sort with the cloud above the
value.  The clouds here sit on the edges of that: empty ones, single points,
every space and maximal dimension next to each other, neighbour lists around
the warp's sort sizes (32 and 256) and beyond them, radii far below and above the
cloud's extent.
"""
import numpy as np
import pytest

from specseqplusplus_b200 import Engine, gen

pytestmark = pytest.mark.gpu


def host(r):
    if r[0] == "lowerstar":
        return gen.lowerstar_from_field(r[1], r[2])
    if len(r[1]) == 0:  # the host builder takes no empty cloud
        return gen.BoundaryMatrix(np.zeros(0, np.int32), np.zeros(1, np.int64), np.zeros(0, np.int32),
                                  np.zeros(0, np.float32))
    return gen.rips_from_points(r[1], r[2], r[3])


def check(requests):
    with Engine(0) as e:
        for _ in range(2):  # the second build reuses the buffers
            e.load_built_batch(requests)
            got = e.input_matrix(values=True)
        n = z = 0
        for i, r in enumerate(requests):
            m = host(r)
            assert np.array_equal(got.dims[n:n + m.ncols], m.dims)
            assert np.array_equal(got.col_ptr[n:n + m.ncols + 1], m.col_ptr + z)
            assert np.array_equal(got.rows[z:z + m.nnz], m.rows + n)
            assert np.array_equal(got.values[n:n + m.ncols].view(np.int32), m.values.view(np.int32))
            assert np.array_equal(e.batch_values(i).view(np.int32), m.values.view(np.int32))
            n += m.ncols
            z += m.nnz
        assert got.ncols == n and got.nnz == z


def cloud(rng, n, d, scale=1.0):
    return (rng.random((n, d), dtype=np.float32) * np.float32(scale)).astype(np.float32)


def test_every_dimension_side_by_side():
    rng = np.random.default_rng(1)
    check([("rips", cloud(rng, 40 + 7 * d, d), 0.3, maxdim) for d in (1, 2, 3) for maxdim in (0, 1, 2, 3)])


@pytest.mark.parametrize("same", [True, False])
def test_empty_and_tiny_clouds(same):
    rng = np.random.default_rng(2)
    sizes = [0, 1, 0, 0, 2, 31, 0, 33, 1, 0]
    check([("rips", cloud(rng, n, 2), 0.4, 2 if same else i % 4) for i, n in enumerate(sizes)])
    check([("rips", cloud(rng, 0, 3), 0.4, 2)] * 3)


@pytest.mark.parametrize("n", [31, 32, 33, 34, 255, 256, 257, 258, 400])
def test_complete_graphs_around_the_sort_sizes(n):
    # point 0's upper list holds n - 1 neighbours; a second cloud follows
    rng = np.random.default_rng(n)
    check([("rips", cloud(rng, n, 2), 2.0, 1), ("rips", cloud(rng, 50, 3), 0.3, 3)])


def test_radii_and_extents():
    rng = np.random.default_rng(3)
    same = np.full((70, 3), 0.25, dtype=np.float32)
    line = np.zeros((90, 3), dtype=np.float32)
    line[:, 1] = np.arange(90) * 1e-3
    check([("rips", cloud(rng, 300, 3), 1e-7, 3), ("rips", cloud(rng, 300, 3, 1e6), 1e3, 3),
           ("rips", same, 0.0, 1), ("rips", line, 1.5e-3, 3), ("rips", -cloud(rng, 120, 3), 0.2, 3),
           ("rips", cloud(rng, 80, 2) + np.float32(1e5), 0.5, 2)])


def test_fields_between_clouds():
    rng = np.random.default_rng(4)
    f = rng.normal(size=(4, 5, 6)).astype(np.float32)
    check([("lowerstar", f, 3), ("rips", cloud(rng, 60, 3), 0.4, 3), ("rips", cloud(rng, 70, 2), 0.3, 2),
           ("lowerstar", f[:1], 2), ("lowerstar", f, 0), ("rips", cloud(rng, 20, 1), 0.1, 1)])


def test_many_clouds():
    rng = np.random.default_rng(5)
    check([("rips", cloud(rng, int(rng.integers(0, 60)), 2 + i % 2), 0.25, 2 + i % 2) for i in range(300)])
