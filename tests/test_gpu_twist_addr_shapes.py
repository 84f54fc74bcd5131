"""The Twist address lane where its sorted order can go wrong, bit for bit
against the oracle: one address bit (no sort pass), one and two and three radix
passes, item counts around a block (256) and a sort tile (2048), every access at
one address (one run over many blocks), accesses at the two ends of the address
space, no events, and gates that are not Boolean."""
import numpy as np
import pytest

import oracle
from memcase import bit_cols, rand_k, to_k
from nightstream_b200 import gpu

pytestmark = pytest.mark.gpu


def columns(kind, ell, A, active, pattern, rng):
    L, P = 1 << ell, 1 << A
    has_r, has_w, ra, wa = (np.zeros(L, np.uint64) for _ in range(4))
    has_r[:active] = rng.random(active) < (0.5 if pattern == "sparse" else 1.0)
    has_w[:active] = rng.random(active) < (0.5 if pattern == "sparse" else 1.0)
    if pattern == "one":
        ra[:active] = wa[:active] = P - 1
    elif pattern == "ends":
        ra[:active], wa[:active] = (rng.integers(0, 2, active) * (P - 1) for _ in range(2))
    else:
        ra[:active], wa[:active] = (rng.integers(0, P, active) for _ in range(2))
    ra, wa = ra * has_r, wa * has_w
    gate = lambda h: np.where(h[:, None] != 0, rand_k(rng, L), 0).astype(np.uint64) if pattern == "sparse" else to_k(h)
    vals = lambda h: np.where(h[:, None] != 0, rand_k(rng, L), 0).astype(np.uint64)
    read = [gate(has_r)[None], vals(has_r)[None], bit_cols(ra, A)]
    write = [gate(has_w)[None], vals(has_w)[None], bit_cols(wa, A)]
    if kind == 0:
        return np.concatenate(read + write)
    return np.concatenate([write[0], vals(has_w)[None], write[1], write[2]])


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("ell,A,active,pattern", [
    (3, 1, 8, "uniform"), (8, 1, 256, "one"), (8, 2, 129, "ends"), (9, 9, 257, "sparse"), (11, 10, 1024, "uniform"),
    (11, 17, 1025, "uniform"), (12, 18, 2500, "ends"), (12, 5, 3000, "one"), (6, 4, 0, "uniform"), (10, 12, 513, "sparse")])
def test_twist_addr_shapes_match_oracle(ctx, kind, ell, A, active, pattern):
    rng = np.random.default_rng(ell * 1000 + A * 10 + kind)
    cols = columns(kind, ell, A, active, pattern, rng)
    r_cycle = rand_k(rng, ell)
    init = [(int(a), tuple(int(x) for x in rand_k(rng, 1)[0])) for a in sorted({0, 1, (1 << A) - 1, (1 << A) // 2})]
    ref = oracle.TwistAddrOracle(kind, cols, r_cycle, A, init)
    g = gpu.GpuTwistAddrOracle(ctx, kind, cols, r_cycle, A, init)
    xs = np.array([[0, 0], [1, 0], [2, 0], [12345, 678]], np.uint64)
    for rnd in range(A + 1):
        assert np.array_equal(g.evals_at(xs), ref.evals_at(xs)), f"round {rnd}"
        if rnd < A:
            r = rand_k(rng, 1)[0]
            g.fold(r)
            ref.fold(r)
    g.close()


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("A,active", [(1, 5), (6, 300), (11, 1000)])
def test_rounds_in_any_call_order(ctx, kind, A, active):
    """Values asked twice, folds without values in between (the order of the next round is
    then not there yet), and a fold as the last call."""
    rng = np.random.default_rng(A * 10 + kind)
    ell = 10
    cols = columns(kind, ell, A, active, "uniform", rng)
    r_cycle = rand_k(rng, ell)
    init = [(int(a), tuple(int(x) for x in rand_k(rng, 1)[0])) for a in sorted({0, (1 << A) - 1})]
    ref = oracle.TwistAddrOracle(kind, cols, r_cycle, A, init)
    g = gpu.GpuTwistAddrOracle(ctx, kind, cols, r_cycle, A, init)
    xs = np.array([[0, 0], [1, 0], [2, 0], [5, 6]], np.uint64)
    for rnd in range(A):
        if rnd % 4 != 1:
            for _ in range(1 + rnd % 3):
                assert np.array_equal(g.evals_at(xs), ref.evals_at(xs)), f"round {rnd}"
        r = rand_k(rng, 1)[0]
        g.fold(r)
        ref.fold(r)
    assert np.array_equal(g.evals_at(xs), ref.evals_at(xs))
    g.close()
