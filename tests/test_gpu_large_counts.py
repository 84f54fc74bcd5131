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
