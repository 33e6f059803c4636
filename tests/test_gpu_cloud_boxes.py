"""Bounding boxes and cell grids of point clouds that several blocks read.

A block takes 2,048 points or more, 512 blocks a cloud at most; the last one makes
the grid.  The points with the outermost coordinates (or with one that is not a
number) stand where a block begins or ends.
"""
import numpy as np
import pytest

from specseqplusplus_b200 import Engine, SsppError, gen
from test_gpu_build_joint import check, cloud

pytestmark = pytest.mark.gpu


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
