"""Counts above the 65535 blocks of a launch's second grid dimension."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
Q = (1 << 64) - (1 << 32) + 1


def test_commitment_of_more_than_65535_vectors(ctx):
    """A separate sequence launch (65 K blocks a CTA, one past the fused form) over 65540 vectors."""
    m, n_vec, rng = 130, 65540, np.random.default_rng(5)
    pp = rng.integers(0, Q, size=(1, m, 54), dtype=np.uint64)
    ctx.pp_upload(pp)
    Z = rng.integers(-1, 2, size=(5, 54, m)).astype(np.int8)
    d = torch.from_numpy(Z).cuda().repeat(n_vec // 5, 1, 1)  # vector v is Z[v % 5]
    out = torch.zeros((n_vec, 1, 54), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ctx.commit_device(d.data_ptr(), n_vec, m, out.data_ptr(), small_digits=True)
    ctx.synchronize()
    want = np.stack([O.commit_digits(pp, z) for z in Z])
    got = out.cpu().numpy().view(np.uint64).reshape(n_vec // 5, 5, 1, 54)
    assert (got == want).all()


def test_bitness_oracle_of_more_than_65535_columns(ctx):
    """2^14 rows: the fold after the first round is a launch of its own, a block row per column."""
    import ctypes

    from memcase import rand_k
    from nightstream_b200 import gpu
    ell, n_cols, rng = 14, 65540, np.random.default_rng(6)
    at = [3, n_cols - 1]  # the columns that are not zero, which add nothing
    vals = rand_k(rng, 2 << ell).reshape(2, 1 << ell, 2)
    w, point = rand_k(rng, n_cols), rand_k(rng, ell)
    cols = torch.zeros((n_cols, 1 << ell, 2), dtype=torch.int64, device="cuda")
    for i, c in enumerate(at):
        cols[c] = torch.from_numpy(vals[i].view(np.int64)).cuda()
    torch.cuda.synchronize()
    claim, h = np.empty(2, np.uint64), ctypes.c_void_p()
    ctx.check(ctx.lib.neo_gpu_mem_oracle_create_device(ctx.h, gpu.MEM_BITNESS, ell, point.ctypes.data, 0, None, None, n_cols,
                                                       cols.data_ptr(), w.ctypes.data, claim.ctypes.data, ctypes.byref(h)))
    ref = O.MemOracle(gpu.MEM_BITNESS, vals, point, None, None, w[at])
    try:
        assert np.array_equal(claim, ref.claim)
        xs = np.array([[x, 0] for x in range(4)], np.uint64)
        ys = np.empty_like(xs)
        for rnd in range(ell + 1):
            ctx.check(ctx.lib.neo_gpu_mem_oracle_evals(h, xs.ctypes.data, len(xs), ys.ctypes.data))
            assert np.array_equal(ys, ref.evals_at(xs)), f"round {rnd}"
            if rnd < ell:
                r = rand_k(rng, 1)[0]
                ctx.check(ctx.lib.neo_gpu_mem_oracle_fold(h, r.ctypes.data))
                ref.fold(r)
    finally:
        ctx.lib.neo_gpu_mem_oracle_destroy(h)
        del cols
        torch.cuda.empty_cache()
