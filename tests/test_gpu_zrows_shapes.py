"""ME outputs on the tensor cores at the edges of their tiles, bit for bit against the
oracle: a last half chunk of columns, row groups with a remainder, one to four vectors,
full-range digits, enough columns for several blocks a row group; and the shapes that
stay with the general kernel (rows not 64-byte aligned, five vectors)."""
import numpy as np
import pytest

import oracle as O
from nightstream_b200 import synth
from nightstream_b200.ccs import CcsStructure, CscMatrix

pytestmark = pytest.mark.gpu
Q = (1 << 64) - (1 << 32) + 1


@pytest.mark.parametrize("m,t,k,lim", [(64, 1, 1, 1), (192, 3, 3, 127), (1024, 4, 5, 127), (128 * 150 + 64, 2, 1, 127),
                                       (1 << 17, 3, 2, 1), (100, 3, 2, 127), (128, 5, 2, 127)])
def test_me_y_shapes(ctx, m, t, k, lim):
    ell = 6
    n = 1 << ell
    rng = np.random.default_rng(m + t)
    mats = []
    for _ in range(t):
        cols = np.concatenate([np.arange(m), rng.integers(0, m, m // 2)])
        mats.append(CscMatrix.from_coo(n, m, rng.integers(0, n, cols.size), cols, rng.integers(0, Q, cols.size, dtype=np.uint64)))
    ccs = CcsStructure(n, m, mats, [(1, [1] + [0] * (t - 1))])
    Z = rng.integers(-lim - (lim > 1), lim + 1, size=(k, 54, m)).astype(np.int8)
    r = synth.uniform_k(rng, ell)
    y, ysc = ctx.me_y(ccs, Z, r)
    for i in range(k):
        y2, ysc2 = O.me_y_at_r(ccs, Z[i], ell, r)
        y1 = y if k == 1 and y.ndim == 3 else y[i]
        s1 = ysc if k == 1 and ysc.ndim == 2 else ysc[i]
        assert np.array_equal(y1, y2) and np.array_equal(s1, ysc2)


@pytest.mark.parametrize("digit", [-128, 127])
def test_me_y_extreme_sums(ctx, digit):
    """Every digit at the end of int8 and every limb near 255: the largest 32-bit sums
    of a block's column range."""
    ell, n, m = 1, 2, 1 << 16
    M = CscMatrix.from_coo(n, m, np.zeros(m, np.int64), np.arange(m), np.full(m, Q - 1, np.uint64))
    ccs = CcsStructure(n, m, [M], [(1, [1])])
    Z = np.full((1, 54, m), digit, np.int8)
    r = np.array([[0, 0]], np.uint64)
    y, ysc = ctx.me_y(ccs, Z, r)
    y2, ysc2 = O.me_y_at_r(ccs, Z[0], ell, r)
    assert np.array_equal(np.asarray(y).reshape(y2.shape), y2) and np.array_equal(np.asarray(ysc).reshape(ysc2.shape), ysc2)
