"""Bounding boxes and cell grids of point clouds that several blocks read.

A block takes 2,048 points or more, 512 blocks a cloud at most; the last one makes
the grid.  The points with the outermost coordinates (or with one that is not a
number) stand where a block begins or ends.
"""
import numpy as np
import pytest

from specseqplusplus_b200 import Engine, SsppError, gen
from specseqplusplus_b200.gen import BoundaryMatrix
import test_gpu_build_joint as joint
from test_gpu_build_joint import cloud

pytestmark = pytest.mark.gpu


def check(requests, vertices=()):
    """test_gpu_build_joint.check; the requests listed are vertices alone (the host builder wants finite points)"""
    of = {id(requests[i]) for i in vertices}

    def host(r):
        n = len(r[1])
        if id(r) in of:
            return BoundaryMatrix(np.zeros(n, np.int32), np.zeros(n + 1, np.int64), np.zeros(0, np.int32),
                                  np.zeros(n, np.float32))
        return ordinary(r)

    ordinary, joint.host = joint.host, host
    try:
        joint.check(requests)
    finally:
        joint.host = ordinary


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4096, 4097, 300_000])
@pytest.mark.parametrize("d", [1, 2, 3])
def test_outliers_at_the_blocks_ends(n, d):
    rng = np.random.default_rng(n + d)
    p = cloud(rng, n, d)
    for i in {0, n - 1, min(2047, n - 1), min(2048, n - 1)}:
        p[i] = rng.uniform(-5, 5, d)
    check([("rips", p, gen.rips_radius_for_degree(n, d, 1.0), min(d, 2))])


def test_uneven_clouds_side_by_side():
    rng = np.random.default_rng(7)
    sizes = [0, 5000, 1, 30_000, 2048, 0, 3, 2049, 100_000]
    check([("rips", cloud(rng, n, 1 + i % 3) - np.float32(0.5), gen.rips_radius_for_degree(max(n, 9), 1 + i % 3, 2.0), 2)
           for i, n in enumerate(sizes)])


@pytest.mark.parametrize("at", [0, 2047, 2048, 99_999])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_a_coordinate_that_is_not_finite(at, value):
    p = gen.points(100_000, 3, 1)
    good = gen.rips_radius_for_degree(100_000, 3, 1.0)
    q = p.copy()
    q[at, 2] = value
    with Engine(0) as e:
        for _ in range(2):
            with pytest.raises(SsppError) as ei:
                e.load_rips(q, good, 2)
            assert ei.value.code == 1 and "non-finite" in str(ei.value)
            e.load_rips(p, good, 2)
            assert e.input_matrix().ncols > 100_000


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 3e38])
def test_points_alone_may_have_any_coordinate(value):
    # without edges (maximal dimension 0) the coordinates are not looked at
    rng = np.random.default_rng(11)
    q = cloud(rng, 5000, 2)
    q[[0, 2048, 4999], 1] = value
    q[17, 0] = -value
    check([("rips", cloud(rng, 60, 3), 0.4, 3), ("rips", q, 0.1, 0), ("rips", q[:0], 0.1, 0),
           ("rips", cloud(rng, 3000, 2), 0.02, 2)], vertices=(1,))
    check([("rips", q, 0.1, 0)] * 2, vertices=(0, 1))
    with Engine(0) as e:
        for _ in range(2):
            e.load_rips(q, 0.1, 0)
            m = e.input_matrix(values=True)
            assert m.ncols == 5000 and m.nnz == 0
            assert not m.dims.any() and not m.col_ptr.any() and not m.values.any()


@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("scale", [1e-24, 1e-22, 1e-21, 3e-20, 1e-18, 1.0])
@pytest.mark.parametrize("radius", [0.0, 1e-30, 2e-23, 4e-23, 3e-22, 9e-20, 1.1e-19])
def test_distances_whose_squares_underflow(d, scale, radius):
    rng = np.random.default_rng(d)
    p = cloud(rng, 36, d, scale)
    q = np.concatenate([cloud(rng, 40, d, scale), cloud(rng, 3, d)])  # and a few far away: larger cells
    check([("rips", p, radius, 1), ("rips", q, radius, 1)])
