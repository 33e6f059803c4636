"""GPU parity of the edge columns' own reduction (a forest of the vertices).

Graphs whose vertex and edge counts sit around the size up to which one block does
all of it, edges with two, one and no vertices, columns of dimension 1 that are too
long for it, edges beside triangles on small and large inputs, and a matrix that is
no chain complex.
"""
import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params, gen
from specseqplusplus_b200.gen import BoundaryMatrix

pytestmark = pytest.mark.gpu


def graph(nv, edges):
    """nv vertices, then one edge per row of `edges` (any number of distinct vertices)."""
    dims = [0] * nv + [1] * len(edges)
    return BoundaryMatrix.from_columns(dims, [[]] * nv + [sorted(map(int, e)) for e in edges])


def check(m, **params):
    ref = oracle.reduce(m)
    with Engine(0) as e:
        e.load_csc(m)
        e.reduce(Params(**params))
        assert np.array_equal(e.pairs(), ref.pairs)
        assert np.array_equal(e.essentials(), ref.essential)


def shape(kind, nv, ne, rng):
    if kind == "path":  # each edge between neighbours, in a random order, twice over
        i = np.concatenate([rng.permutation(nv - 1)] * (ne // (nv - 1) + 1))[:ne]
        return np.stack([i, i + 1], axis=1)
    if kind == "descending":  # every edge takes the row of the ones before it
        i = nv - 2 - np.arange(ne) % (nv - 1)
        return np.stack([i, np.full(ne, nv - 1)], axis=1)
    if kind == "star":
        return np.stack([np.zeros(ne, int), 1 + rng.integers(0, nv - 1, ne)], axis=1)
    a = rng.integers(0, nv, ne)
    return np.stack([a, (a + 1 + rng.integers(0, nv - 1, ne)) % nv], axis=1)


@pytest.mark.parametrize("kind", ["path", "descending", "star", "random"])
@pytest.mark.parametrize("nv,ne", [(2, 1), (2, 40), (33, 32), (700, 1400), (3000, 5000), (3000, 5191), (3000, 5192),
                                   (3000, 5193), (3000, 9000), (20000, 30000)])
@pytest.mark.parametrize("dualize", [0, 2])
def test_graphs(kind, nv, ne, dualize):
    if dualize and kind in ("star", "descending") and ne > 10000:
        pytest.skip("one vertex column of the dual is as long as the list of edges")
    check(graph(nv, shape(kind, nv, ne, np.random.default_rng(nv + ne))), dualize=dualize)


@pytest.mark.parametrize("nv", [1, 5, 300, 9000])
def test_edges_with_fewer_vertices(nv):
    # relative complexes: an edge into the part taken out has one vertex, or none
    rng = np.random.default_rng(nv)
    edges = [rng.choice(nv, size=min(nv, k), replace=False) for k in rng.integers(0, 3, 2 * nv)]
    check(graph(nv, edges))


@pytest.mark.parametrize("where", [0, 100, 399])
def test_a_longer_column_of_dimension_one(where):
    rng = np.random.default_rng(where)
    edges = [rng.choice(300, size=2, replace=False) for _ in range(400)]
    edges[where] = rng.choice(300, size=3, replace=False)
    check(graph(300, edges))


@pytest.mark.parametrize("grid", [7, 17, 22])
def test_edges_beside_triangles(grid):
    m = gen.lowerstar(grid, 2.0, grid)  # 17: below the size from which dimensions overlap, 22: above
    out = []
    with Engine(0) as e:
        e.load_csc(m)
        for schedule in (1, 2, 1):
            e.reduce(Params(schedule=schedule))
            out.append((e.pairs().copy(), e.essentials().copy()))
    for pairs, ess in out[1:]:
        assert np.array_equal(pairs, out[0][0]) and np.array_equal(ess, out[0][1])


@pytest.mark.parametrize("more", [0, 9000, 140000])
def test_an_edge_that_would_own_and_be_owned(more):
    # the last triangle's boundary is edges 6 and 7, whose boundary is not zero: reduced,
    # it claims edge 6, which counts as positive then and does not claim vertex 2
    dims = [0, 0, 0, 0, 1, 1, 1, 1, 2, 2] + [0] * more
    cols = [[], [], [], [], [0, 1], [2, 3], [1, 2], [0, 1], [4, 7], [6, 7]] + [[]] * more
    with Engine(0) as e:
        e.load_csc(BoundaryMatrix.from_columns(dims, cols))
        for _ in range(2):
            e.reduce(Params())
            assert e.pairs().tolist() == [[1, 4], [3, 5], [6, 9], [7, 8]]
            assert e.essentials().tolist() == [0, 2] + list(range(10, 10 + more))
