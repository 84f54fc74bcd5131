"""The tensor-core commitment at the edges of its shapes, bit for bit against the
oracle: odd and tiny column counts (the last K block's zero column), every
vector-group size with a padded last group, K splits below and above the ring
depths, both sides of the fused / separate sequence rule (12 vectors: 64 and 65
K blocks per CTA), a partial last 128-column block of the sequence launch, and
digits that leave the small-digit form where the call must still be exact."""
import numpy as np
import pytest

import oracle as O
from nightstream_b200 import gpu

pytestmark = pytest.mark.gpu
Q = (1 << 64) - (1 << 32) + 1


def _commit_device(ctx, Z, small):
    import torch
    n_vec, _, m = Z.shape
    d = torch.from_numpy(Z).cuda()
    out = torch.zeros((n_vec, ctx.kappa, 54), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ctx.commit_device(d.data_ptr(), n_vec, m, out.data_ptr(), small_digits=small)
    ctx.synchronize()
    return out.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("m,n_vec,kappa", [(1, 1, 16), (3, 2, 16), (17, 3, 16), (129, 1, 5), (1001, 2, 16), (1026, 5, 16),
                                           (5001, 1, 16), (4099, 7, 16), (12544, 12, 16), (12546, 12, 16), (12549, 9, 16)])
def test_commit_shapes_match_oracle(ctx, m, n_vec, kappa):
    rng = np.random.default_rng(m * 31 + n_vec)
    pp = rng.integers(0, Q, size=(kappa, m, 54), dtype=np.uint64)
    ctx.pp_upload(pp)
    tern = rng.integers(-1, 2, size=(n_vec, 54, m)).astype(np.int8)
    wide = rng.integers(-128, 128, size=(n_vec, 54, m)).astype(np.int8)
    want_t = np.stack([O.commit_digits(pp, z) for z in tern])
    want_w = np.stack([O.commit_digits(pp, z) for z in wide])
    for _ in range(2):  # twice: the accumulators are left zero
        assert np.array_equal(_commit_device(ctx, tern, True), want_t)
        assert np.array_equal(_commit_device(ctx, wide, False), want_w)
    assert np.array_equal(ctx.commit(tern), want_t)
    assert np.array_equal(ctx.commit(wide), want_w)  # host call: checked, redone in the general form


def test_odd_size_with_large_digits_stays_exact(ctx):
    """The small-digit promise broken at an odd column count gives the exact
    result (no error), as the CUDA-core path that served odd counts did."""
    m = 1025
    rng = np.random.default_rng(5)
    pp = rng.integers(0, Q, size=(16, m, 54), dtype=np.uint64)
    ctx.pp_upload(pp)
    Z = rng.integers(-128, 128, size=(2, 54, m)).astype(np.int8)
    assert np.array_equal(_commit_device(ctx, Z, True), np.stack([O.commit_digits(pp, z) for z in Z]))
    Z[0, 3, m - 1] = -128
    assert np.array_equal(ctx.commit(Z), np.stack([O.commit_digits(pp, z) for z in Z]))


def test_small_promise_broken_by_one_digit_is_reported(ctx):
    m = 64
    rng = np.random.default_rng(6)
    ctx.pp_upload(rng.integers(0, Q, size=(16, m, 54), dtype=np.uint64))
    for row, value in ((0, -128), (53, -128)):
        Z = rng.integers(-1, 2, size=(5, 54, m)).astype(np.int8)
        Z[4, row, m - 1] = value
        with pytest.raises(gpu.NeoGpuError) as e:
            _commit_device(ctx, Z, True)
        assert e.value.code == 3
