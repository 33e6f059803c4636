"""GPU parity at limits that ordinary inputs do not reach.

A tile of the one-pass scan that its predecessors do not answer in time takes
their values itself.  That never happens by itself in a test, so the library is
built here with a limit of one poll: every tile that is not answered at once does it.
And point clouds are built together up to 2^26 columns; here up to 20,000, so that
batches are built in several parts.  The allocation-free call's array holds 2^20 ints
instead of 2^24, so that matrices whose fill-in can be counted here end on either side
of its room.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params, SsppError, gen

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _rips(npts, dim, degree, seed):
    pts = gen.points(npts, dim, seed)
    r = gen.rips_radius_for_degree(npts, dim, degree)
    return pts, r, gen.rips(npts, dim, seed, r, dim)


def check_built(e):
    for npts, dim, degree in ((1500, 2, 9.0), (5000, 3, 8.0), (9000, 2, 20.0)):
        pts, r, m = _rips(npts, dim, degree, 5)
        e.load_rips(pts, r, dim)
        got = e.input_matrix()
        for a, b in ((got.dims, m.dims), (got.col_ptr, m.col_ptr), (got.rows, m.rows)):
            assert np.array_equal(a, b), (npts, dim)


def check_reduced(e):
    for m in (_rips(3000, 3, 12.0, 7)[2], gen.lowerstar(17, 1.5, 3), gen.lowerstar(26, 1.5, 4)):
        want = oracle.reduce(m)
        for p in (Params(), Params(dualize=1), Params(dualize=2), Params(model=1, max_iteration=10)):
            e.load_csc(m)
            e.reduce(p)
            assert np.array_equal(e.pairs(), want.pairs), (m.ncols, p)
            assert np.array_equal(e.essentials(), want.essential), (m.ncols, p)
    m = gen.rips(4000, 3, 2, gen.rips_radius_for_degree(4000, 3, 3.0), 3)
    p = Params(model=3, max_iteration=100)
    e.load_csc(m)
    e.reduce(p)
    want = oracle.reduce(m, model=3, max_iteration=100)
    assert np.array_equal(e.pairs(), want.pairs) and np.array_equal(e.essentials(), want.essential)


def check_split(e):
    import test_gpu_build_joint as joint

    rng = np.random.default_rng(9)

    def rips(n, d, degree, maxdim):
        return ("rips", joint.cloud(rng, n, d), gen.rips_radius_for_degree(max(n, 2), d, degree), maxdim)

    field = ("lowerstar", rng.normal(size=(5, 6, 7)).astype(np.float32), 3)
    small = [rips(int(rng.integers(0, 400)), 2 + i % 2, 8.0, 2 + i % 2) for i in range(40)]
    joint.check(small)
    # one larger than the limit by itself, first, last and in the middle; parts that end at a field
    large = rips(3000, 3, 14.0, 3)
    joint.check([large] + small[:5] + [large, field] + small[5:9] + [rips(0, 2, 1.0, 2), large])
    joint.check([large, large, large])
    joint.check([rips(1500, 2, 9.0, i % 4) for i in range(9)])
    # the batch's columns are those of its members, wherever the parts ended
    requests = small[:20] + [field] + small[20:]
    e.load_built_batch(requests)
    e.reduce(Params())
    for r, (pairs, ess) in zip(requests, e.batch_results(), strict=True):
        m = joint.host(r)
        want = oracle.reduce(m)
        assert np.array_equal(pairs, want.pairs) and np.array_equal(ess, want.essential)


def check_fill(e):
    import torch
    from test_gpu_noalloc_buffers import fill_in
    from test_zz_no_alloc import _noalloc_pairs

    def left(m):  # room for fill-in that a column-after-column reduction leaves
        took, room = fill_in(m)
        return room - (16 << 20) + (1 << 20) - took

    def first(m, n):
        return gen.BoundaryMatrix(m.dims[:n], m.col_ptr[:n + 1], m.rows[:m.col_ptr[n]])

    for npts, dim, degree in ((400, 2, 26.0), (150, 2, 40.0), (200, 2, 40.0)):
        m = gen.rips(npts, dim, 3, gen.rips_radius_for_degree(npts, dim, degree), dim)
        lo, hi = 1000, m.ncols  # the subcomplex of the first lo columns fits, that of the first hi does not
        assert left(m) < 0 <= left(first(m, lo))
        while hi - lo > 1:
            n = (lo + hi) // 2
            lo, hi = (n, hi) if left(first(m, n)) >= 0 else (lo, n)
        for _ in range(2):
            assert np.array_equal(_noalloc_pairs(first(m, lo), torch), oracle.reduce(first(m, lo)).pairs)
            with pytest.raises(SsppError) as ei:
                _noalloc_pairs(first(m, hi), torch)
            assert ei.value.code == 2


def main(lib, check):
    from specseqplusplus_b200 import engine

    engine.LIB_PATH = lib
    with Engine(0) as e:
        for _ in range(1 if check == "check_fill" else 3):
            globals()[check](e)


@pytest.fixture(scope="module")
def limited(tmp_path_factory):
    sys.path.insert(0, os.path.join(ROOT, "specseqplusplus_b200"))
    import build

    d = tmp_path_factory.mktemp("limited")
    lib = str(d / "libsspp.so")
    build.build_engine(lib, str(d / "obj"), ["-DSSPP_SCAN_POLLS=1", "-DSSPP_MAX_JOINT_COLS=20000",
                                           "-DSSPP_SCRATCH_INTS=(1<<20)"])
    return lib


@pytest.mark.gpu
@pytest.mark.parametrize("check", ["check_built", "check_reduced", "check_split", "check_fill"])
def test_with_small_limits(limited, check):
    code = "import sys, test_gpu_limits as t; t.main(sys.argv[1], sys.argv[2])"
    path = os.pathsep.join([ROOT, os.path.join(ROOT, "oracle"), os.path.join(ROOT, "tests")])
    r = subprocess.run([sys.executable, "-c", code, limited, check], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=path))
    assert r.returncode == 0, r.stdout + r.stderr
