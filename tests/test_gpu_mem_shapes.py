"""Time-lane oracles at the edges of the evaluation launch's shapes, every round
bit for bit against the oracle: one pair, 16 and 17 pairs (one block per point /
tiles), a size whose fold is a launch of its own, degrees from 2 to 31 (one to
eight warps a point set, more points than warps), few and many bitness columns
(several factor chunks), sparse and dense gates, and factors that are zero."""
import numpy as np
import pytest

import oracle
from memcase import rand_k
from nightstream_b200 import gpu

pytestmark = pytest.mark.gpu


def _rounds(ctx, kind, cols, r_point, weights, ell, rng, r_addr=None, init=None, some=None):
    ref = oracle.MemOracle(kind, cols, r_point, r_addr, init, weights)
    g = gpu.GpuMemOracle(ctx, kind, cols, r_point, r_addr, init, weights)
    assert np.array_equal(g.claim, ref.claim)
    xs = np.array([[x, 0] for x in range(g.degree_bound() + 1)] + [[99, 7]], np.uint64)
    for rnd in range(ell + 1):
        got = g.evals_at(xs)
        assert np.array_equal(got, ref.evals_at(xs)), f"round {rnd}"
        assert np.array_equal(g.evals_at(xs[::-1]), got[::-1])  # asked twice
        if rnd < ell:
            r = rand_k(rng, 1)[0]
            g.fold(r)
            ref.fold(r)
            if rnd == 1 and ell > 3:  # two folds without an evaluation between
                r = rand_k(rng, 1)[0]
                g.fold(r)
                ref.fold(r)
                break
    if ell > 3:
        assert np.array_equal(g.evals_at(xs), ref.evals_at(xs))
    for rnd in range(g.num_rounds()):
        r = rand_k(rng, 1)[0]
        g.fold(r)
        ref.fold(r)
        assert np.array_equal(g.evals_at(xs), ref.evals_at(xs)), f"late round {rnd}"
    g.close()


@pytest.mark.parametrize("ell,n_cols,density", [(1, 1, 1.0), (2, 3, 1.0), (5, 31, 1.0), (6, 2, 0.1), (7, 18, 0.5), (9, 9, 0.02),
                                                (10, 5, 0.0), (13, 4, 0.01), (14, 2, 1.0)])
def test_product_shapes(ctx, ell, n_cols, density):
    rng = np.random.default_rng(ell * 100 + n_cols)
    L = 1 << ell
    cols = rand_k(rng, n_cols * L).reshape(n_cols, L, 2)
    cols[min(1, n_cols - 1)][rng.random(L) >= density] = 0
    _rounds(ctx, gpu.MEM_PRODUCT, cols, None, None, ell, rng)


@pytest.mark.parametrize("ell,n_cols,density", [(1, 1, 1.0), (4, 0, 1.0), (5, 40, 0.3), (6, 70, 1.0), (8, 16, 0.05), (13, 3, 0.01)])
def test_bitness_shapes(ctx, ell, n_cols, density):
    rng = np.random.default_rng(ell * 100 + n_cols)
    L = 1 << ell
    cols = rand_k(rng, n_cols * L).reshape(n_cols, L, 2)
    cols[:, rng.random(L) >= density] = 0
    _rounds(ctx, gpu.MEM_BITNESS, cols, rand_k(rng, ell), rand_k(rng, max(1, n_cols)), ell, rng)


@pytest.mark.parametrize("kind,A", [(gpu.MEM_TWIST_READ, 1), (gpu.MEM_TWIST_WRITE, 28), (gpu.MEM_VAL_EVAL, 20)])
def test_twist_degrees(ctx, kind, A):
    ell = 7
    rng = np.random.default_rng(kind * 10 + A)
    n_cols = {gpu.MEM_TWIST_READ: 4 + 2 * A, gpu.MEM_TWIST_WRITE: 3 + A, gpu.MEM_VAL_EVAL: 2 + A}[kind]
    cols = rand_k(rng, n_cols << ell).reshape(n_cols, 1 << ell, 2)
    init = rand_k(rng, 1)[0] if kind != gpu.MEM_VAL_EVAL else None
    _rounds(ctx, kind, cols, rand_k(rng, ell), None, ell, rng, rand_k(rng, A), init)
