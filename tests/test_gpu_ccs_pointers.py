"""Column pointers and matrix offsets of an uploaded CCS are checked before any launch: the
device forms its indexes from them (both uploads: with the row copy and without)."""
import numpy as np
import pytest

import oracle as O
from nightstream_b200 import gpu, synth
from nightstream_b200.ccs import CcsStructure, CscMatrix

pytestmark = pytest.mark.gpu
Q = (1 << 64) - (1 << 32) + 1
ELL = 4
N = 1 << ELL


def _ccs(seed, change=None):
    """[I, A, B, C] with `change` applied to the description's col_ptr [t][n + 1] and nnz_off [t + 1]."""
    rng = np.random.default_rng(seed)
    mats = [None] + [CscMatrix.from_coo(N, N, rng.integers(0, N, 3 * N), rng.integers(0, N, 3 * N),
                                        rng.integers(0, Q, 3 * N, dtype=np.uint64)) for _ in range(3)]
    ccs = CcsStructure(N, N, mats, [(1, [0, 1, 1, 0]), (Q - 1, [0, 0, 0, 1])])
    if change:
        d = ccs.desc()
        change(d._keep[1], d._keep[2])
        ccs.desc = lambda: d
    return ccs


def _args(ccs, k=2):
    rng = np.random.default_rng(3)
    Z = rng.integers(-1, 2, size=(k, 54, N)).astype(np.int8)
    return (ccs, Z, 2, synth.uniform_k(rng, 6), synth.uniform_k(rng, 6), synth.uniform_k(rng, ELL),
            synth.uniform_k(rng, 1)[0], synth.uniform_k(rng, ELL), 6, ELL, 6)


def _twice(cp, off):      # columns 0 and 2 would both take every entry
    cp[1, :] = cp[1, N]
    cp[1, 0] = cp[1, 2] = 0


def _above(cp, off):      # an inner pointer past the matrix
    cp[2, 5] = 3 * N + 7


def _offsets(cp, off):    # matrix 2 begins after its end
    off[2] = off[3] + 1


def _past(cp, off):       # matrix 2 ends past the nonzeros
    off[3] = off[4] + 5
    cp[2, N] = off[3] - off[2]


@pytest.mark.parametrize("change", [_twice, _above, _offsets, _past])
def test_bad_pointers_are_refused(ctx, change):
    args = _args(_ccs(1, change))
    for call in (lambda: gpu.GpuCcsOracle(ctx, *args), lambda: ctx.me_y(args[0], args[1], args[5])):
        with pytest.raises(gpu.NeoGpuError) as e:
            call()
        assert e.value.code == 1
    ok = _args(_ccs(1))  # the context still works
    g, o = gpu.GpuCcsOracle(ctx, *ok), O.CcsOracle(*ok)
    xs = np.array([[x, 0] for x in range(7)], np.uint64)
    assert np.array_equal(g.evals_at(xs), o.evals_at(xs))
    g.close()


def test_entries_before_the_first_column_belong_to_none(ctx):
    """col_ptr[0] > 0: the matrix is the one without its first entries."""
    full = _ccs(2)
    M = full.matrices[1]
    skip = int(M.col_ptr[2])  # the entries of columns 0 and 1
    cut = _ccs(2)
    cut.matrices[1] = CscMatrix(N, N, np.maximum(M.col_ptr, np.uint64(skip)) - np.uint64(skip), M.row_idx[skip:], M.vals[skip:])

    def late(cp, off):
        cp[1, :2] = skip
    a, b = _args(_ccs(2, late)), _args(cut)
    g, o = gpu.GpuCcsOracle(ctx, *a), O.CcsOracle(*b)
    xs = np.array([[x, 0] for x in range(7)], np.uint64)
    rng = np.random.default_rng(4)
    for rnd in range(ELL + 6):
        assert np.array_equal(g.evals_at(xs), o.evals_at(xs)), f"round {rnd}"
        r = synth.uniform_k(rng, 1)[0]
        g.fold(r)
        o.fold(r)
    for x, y in zip(g.me_outputs(), o.me_outputs()):
        assert np.array_equal(x, y)
    g.close()
    for x, y in zip(ctx.me_y(a[0], a[1], a[5]), ctx.me_y(b[0], b[1], b[5])):
        assert np.array_equal(x, y)
