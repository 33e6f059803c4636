"""GPU parity of reductions that stop at a band and go on in a later block.

Spectral-sequence blocks are schedule 2's: a column whose lowest row drops below its
block's band parks and is taken up again, in rounds that stop there.  The matrices are
those of the rounds' and the dual's tests, block sizes from one column to all.
"""
import numpy as np
import pytest

import oracle
from helpers import random_complex
from specseqplusplus_b200 import Engine, Params, gen
from test_gpu_rounds import LENGTHS, check, matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,l1,l2", [(128, 32, 96), (256, 32, 8192), (256, 64, 8000)])
@pytest.mark.parametrize("block,growth", [(50, 1.0), (700, 1.3), (1 << 30, 1.0)])
def test_long_columns_over_short_owners(threads, l1, l2, block, growth):
    rng = np.random.default_rng(7)
    n = 2000
    cols = [[r] + list(rng.integers(max(0, r - 60), r, size=rng.integers(0, 5))) for r in range(8, n) if r % 7]
    rng.shuffle(cols)
    for length in LENGTHS[:-1]:
        cols.append(rng.choice(n, size=length, replace=False))
        cols.append(np.arange(n - length, n))
    check(matrix(n, cols), Params(schedule=2, level1_capacity=l1, level2_capacity=l2, heavy_threads=threads,
                                  ss_block_size=block, growth=growth))


@pytest.mark.parametrize("length", [1, 4, 5, 31, 32, 33, 64])
@pytest.mark.parametrize("block", [1, 60, 200])
def test_owners_of_every_addend_length(length, block):
    rng = np.random.default_rng(length)
    n = 500
    cols = [np.append(rng.choice(r, size=length - 1, replace=False), r) for r in range(length, n)]
    cols += [rng.choice(n, size=k, replace=False) for k in (3, 17, 32, 33, 100, 256, 300, 450)]
    check(matrix(n, cols), Params(schedule=2, level1_capacity=64, ss_block_size=block, growth=1.0))


@pytest.mark.parametrize("seed", range(6))
def test_random_matrices(seed):
    rng = np.random.default_rng(100 + seed)
    n = int(rng.integers(20, 600))
    cols = [rng.choice(n, size=int(rng.integers(1, min(n, 40))), replace=False) for _ in range(2 * n)]
    for l1, l2 in ((32, 32), (32, 128), (64, 4096)):
        check(matrix(n, cols), Params(schedule=2, level1_capacity=l1, level2_capacity=l2,
                                      ss_block_size=1 + 97 * seed, growth=1.2))


@pytest.mark.parametrize("dualize", [0, 1, 2])
@pytest.mark.parametrize("block,growth", [(3, 1.1), (64, 1.0), (1000, 2.0)])
def test_complexes(dualize, block, growth):
    rng = np.random.default_rng(dualize)
    mats = [random_complex(rng, 9, 0.6, 3), gen.rips(400, 3, 5, 0.2, 3), gen.rips(600, 2, 6, 0.08, 2),
            gen.lowerstar(9, 1.5, 3)]
    p = Params(schedule=2, dualize=dualize, ss_block_size=block, growth=growth, level1_capacity=32)
    with Engine(0) as e:
        for m in mats:
            ref = oracle.reduce(m)
            e.load_csc(m)
            e.reduce(p)
            assert np.array_equal(e.pairs(), ref.pairs)
            assert np.array_equal(e.essentials(), ref.essential)
        e.load_batch(mats)
        e.reduce(p)
        for m, (pairs, ess) in zip(mats, e.batch_results(), strict=True):
            ref = oracle.reduce(m)
            assert np.array_equal(pairs, ref.pairs) and np.array_equal(ess, ref.essential)
