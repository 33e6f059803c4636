"""GPU parity when the scans' tiles do not wait for one another.

A tile of the one-pass scan that its predecessors do not answer in time takes
their values itself.  That never happens by itself in a test, so the library is
built here with a limit of one poll: every tile that is not answered at once does it.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from specseqplusplus_b200 import Engine, Params, gen

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


def main(lib, check):
    from specseqplusplus_b200 import engine

    engine.LIB_PATH = lib
    with Engine(0) as e:
        for _ in range(3):
            globals()[check](e)


@pytest.fixture(scope="module")
def impatient(tmp_path_factory):
    sys.path.insert(0, os.path.join(ROOT, "specseqplusplus_b200"))
    import build

    d = tmp_path_factory.mktemp("impatient")
    lib = str(d / "libsspp.so")
    build.build_engine(lib, str(d / "obj"), ["-DSSPP_SCAN_POLLS=1"])
    return lib


@pytest.mark.gpu
@pytest.mark.parametrize("check", ["check_built", "check_reduced"])
def test_tiles_that_take_the_earlier_values_themselves(impatient, check):
    code = "import sys, test_gpu_scan_waits as t; t.main(sys.argv[1], sys.argv[2])"
    path = os.pathsep.join([ROOT, os.path.join(ROOT, "oracle"), os.path.join(ROOT, "tests")])
    r = subprocess.run([sys.executable, "-c", code, impatient, check], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=path))
    assert r.returncode == 0, r.stdout + r.stderr
