"""Public parameters of an odd column count whose tensor-core tiles do not fit the device: the
upload succeeds and commitments run on the CUDA cores."""
import numpy as np
import pytest

import oracle as O
from nightstream_b200 import gpu

pytestmark = pytest.mark.gpu
Q = (1 << 64) - (1 << 32) + 1


def test_odd_column_count_without_room_for_tiles():
    import torch
    m = 60001  # 492 MB of tiles, 26 MB of public parameters
    rng = np.random.default_rng(8)
    pp = rng.integers(0, Q, size=(1, m, 54), dtype=np.uint64)
    Z = rng.integers(-1, 2, size=(54, m)).astype(np.int8)
    c = gpu.Context(0)
    small = rng.integers(0, Q, size=(1, 33, 54), dtype=np.uint64)
    c.pp_upload(small)  # the upload's and the commitment's kernels are loaded before memory gets short
    assert np.array_equal(c.commit(Z[:, :33].copy()), O.commit_digits(small, Z[:, :33].copy()))
    c.synchronize()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8, device="cuda")
    try:
        c.pp_upload(pp)
        short = c.commit(Z)
    finally:
        del fill
        torch.cuda.empty_cache()
    want = O.commit_digits(pp, Z)
    assert np.array_equal(short, want)
    c.pp_upload(pp)  # with room again: the tiles
    assert np.array_equal(c.commit(Z), want)
    c.close()
