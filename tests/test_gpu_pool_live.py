"""What a context's pool keeps is bounded by what is unused, however much is alive, and a
destruction gives the rest back itself."""
import numpy as np
import pytest

from nightstream_b200 import gpu

pytestmark = pytest.mark.gpu
KEEP = 1 << 30
SLACK = 256 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _oracle(c, n_cols):  # 64 MB a column, and half of that for the folded tables
    return gpu.GpuMemOracle(c, gpu.MEM_PRODUCT, np.zeros((n_cols, 1 << 22, 2), np.uint64))


def test_idle_buffers_stay_beside_live_ones():
    c = gpu.Context(0)
    live = _oracle(c, 20)  # 2 GB
    before = _free()
    _oracle(c, 6).close()  # 0.6 GB
    c.synchronize()
    assert _free() < before - (400 << 20)
    _oracle(c, 20).close()  # 2 GB: over the bound
    assert _free() >= before - KEEP - SLACK
    live.close()
    c.close()


def test_destruction_gives_back_before_it_returns():
    c = gpu.Context(0)
    before = _free()
    o = _oracle(c, 20)
    import torch
    o.close()
    now = torch.cuda.mem_get_info()[0]  # with no synchronization in between
    assert now >= before - KEEP - SLACK
    c.close()
    assert _free() >= before - SLACK
