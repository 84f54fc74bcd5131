"""Pi_CCS oracles on matrices that a transposition can get wrong, every round and
the ME outputs bit for bit against the oracle: empty rows and columns, one row
that holds most entries, a matrix without entries, unsorted column order and
repeated (row, column) entries, and an f of degree above the R1CS one (more
coefficients per round record)."""
import numpy as np
import pytest

import oracle as O
from nightstream_b200 import gpu, synth
from nightstream_b200.ccs import CcsStructure, CscMatrix

pytestmark = pytest.mark.gpu
Q = (1 << 64) - (1 << 32) + 1


def _matrix(rng, n, kind):
    if kind == "empty":
        return CscMatrix(n, n, np.zeros(n + 1, np.uint64), np.zeros(0, np.uint32), np.zeros(0, np.uint64))
    nnz = 3 * n
    rows = rng.integers(0, n, nnz)
    cols = rng.integers(0, n // 2 if kind == "skew" else n, nnz)
    if kind == "skew":
        rows[: 2 * n] = n - 1
    M = CscMatrix.from_coo(n, n, rows, cols, rng.integers(0, Q, nnz, dtype=np.uint64))
    for c in range(0, n, 3):  # entries of a column in any order
        a, b = int(M.col_ptr[c]), int(M.col_ptr[c + 1])
        p = rng.permutation(b - a)
        M.row_idx[a:b], M.vals[a:b] = M.row_idx[a:b][p], M.vals[a:b][p]
    return M


@pytest.mark.parametrize("ell,k,kinds,terms", [
    (4, 2, ("skew", "empty", "uniform"), [(1, [0, 1, 1, 0]), (Q - 1, [0, 0, 0, 1])]),
    (7, 3, ("skew", "uniform", "skew"), [(5, [0, 3, 2, 0]), (7, [0, 0, 1, 1]), (Q - 2, [0, 1, 0, 0])]),
    (9, 1, ("uniform", "skew", "empty"), [(1, [1, 1, 0, 0]), (3, [0, 0, 2, 1])]),
])
@pytest.mark.parametrize("wide", [False, True])
def test_ccs_shapes_match_oracle(ctx, ell, k, kinds, terms, wide):
    n = 1 << ell
    rng = np.random.default_rng(ell * 10 + k)
    ccs = CcsStructure(n, n, [None] + [_matrix(rng, n, kd) for kd in kinds], terms)
    lim = 5 if wide else 1
    Z = rng.integers(-lim, lim + 1, size=(k, 54, n)).astype(np.int8)
    d_sc = max(ccs.f_degree + 1, 6)
    args = (ccs, Z, 2, synth.uniform_k(rng, 6), synth.uniform_k(rng, 6), synth.uniform_k(rng, ell),
            synth.uniform_k(rng, 1)[0], synth.uniform_k(rng, ell) if k > 1 else None, 6, ell, d_sc)
    g, o = gpu.GpuCcsOracle(ctx, *args), O.CcsOracle(*args)
    xs = np.array([[x, 0] for x in range(d_sc + 1)], np.uint64)
    for rnd in range(ell + 6):
        assert np.array_equal(g.evals_at(xs), o.evals_at(xs)), f"round {rnd}"
        r = synth.uniform_k(rng, 1)[0]
        g.fold(r)
        o.fold(r)
    for a, b in zip(g.me_outputs(), o.me_outputs()):
        assert np.array_equal(a, b)
    g.close()


def test_identity_without_entries_and_bad_rows(ctx):
    """An identity matrix's ranges are not read; a row index out of range is refused."""
    ccs, z = synth.make_r1cs(4, 3)
    Z = ctx.decomp_b2(z)
    r = synth.uniform_k(np.random.default_rng(1), 4)
    y, _ = ctx.me_y(ccs, Z, r)
    assert y.shape == (4, 54, 2)
    ccs.matrices[2].row_idx[5] = 16
    with pytest.raises(gpu.NeoGpuError) as e:
        ctx.me_y(ccs, Z, r)
    assert e.value.code == 1


@pytest.mark.parametrize("ell_d,k,inputs", [(7, 2, True), (8, 1, False), (8, 3, True), (6, 18, True), (6, 5, False)])
def test_ajtai_rounds_shapes(ctx, ell_d, k, inputs):
    """Ajtai rounds on padded coordinate cubes (folds longer than a warp, rounds past
    the 54 entries), at the largest k of the phase and with one to sixteen points."""
    ell = 4
    n = 1 << ell
    rng = np.random.default_rng(ell_d * 10 + k)
    ccs = CcsStructure(n, n, [None] + [_matrix(rng, n, kd) for kd in ("uniform", "skew", "empty")],
                       [(1, [0, 1, 1, 0]), (3, [2, 0, 0, 1])])
    Z = rng.integers(-1, 2, size=(k, 54, n)).astype(np.int8)
    d_sc = 6
    args = (ccs, Z, 2, synth.uniform_k(rng, ell_d), synth.uniform_k(rng, ell_d), synth.uniform_k(rng, ell),
            synth.uniform_k(rng, 1)[0], synth.uniform_k(rng, ell) if inputs else None, ell_d, ell, d_sc)
    g, o = gpu.GpuCcsOracle(ctx, *args), O.CcsOracle(*args)
    for rnd in range(ell + ell_d):
        xs = synth.uniform_k(rng, 16 if rnd % 2 else 1 + rnd % 5)
        assert np.array_equal(g.evals_at(xs), o.evals_at(xs)), f"round {rnd}"
        r = synth.uniform_k(rng, 1)[0]
        g.fold(r)
        o.fold(r)
    g.close()


def test_row_rounds_across_the_pair_forms(ctx):
    """2^14 rows: the first row round has a thread per pair, the next ones eight lanes;
    an f of degree 7, the largest, fills every coefficient lane."""
    ell, k = 14, 2
    n = 1 << ell
    rng = np.random.default_rng(14)
    ccs = CcsStructure(n, n, [None] + [_matrix(rng, n, kd) for kd in ("uniform", "skew")],
                       [(1, [3, 3, 1]), (Q - 5, [0, 1, 0]), (9, [1, 0, 1])])
    Z = rng.integers(-1, 2, size=(k, 54, n)).astype(np.int8)
    d_sc = ccs.f_degree + 1
    args = (ccs, Z, 2, synth.uniform_k(rng, 6), synth.uniform_k(rng, 6), synth.uniform_k(rng, ell),
            synth.uniform_k(rng, 1)[0], synth.uniform_k(rng, ell), 6, ell, d_sc)
    g, o = gpu.GpuCcsOracle(ctx, *args), O.CcsOracle(*args)
    xs = np.array([[x, 0] for x in range(d_sc + 1)], np.uint64)
    for rnd in range(ell):
        assert np.array_equal(g.evals_at(xs), o.evals_at(xs)), f"round {rnd}"
        r = synth.uniform_k(rng, 1)[0]
        g.fold(r)
        o.fold(r)
    g.close()


@pytest.mark.parametrize("order", ["MIM", "IMMI", "MMI", "IIM"])
def test_identities_between_matrices(ctx, order):
    """The column pointers go up in one copy per run of matrices."""
    ell = 6
    n = 1 << ell
    rng = np.random.default_rng(len(order))
    ccs = CcsStructure(n, n, [None if c == "I" else _matrix(rng, n, "uniform") for c in order], [(1, [1] * len(order))])
    Z = rng.integers(-1, 2, size=(54, n)).astype(np.int8)
    r = synth.uniform_k(rng, ell)
    for a, b in zip(ctx.me_y(ccs, Z, r), O.me_y_at_r(ccs, Z, ell, r)):
        assert np.array_equal(a, b)
