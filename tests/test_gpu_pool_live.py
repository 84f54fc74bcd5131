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


@pytest.mark.parametrize("who", ["context", "torch"])
def test_others_can_have_what_a_destroyed_oracle_used(who):
    """Memory is short; the first context has destroyed an oracle of 0.9 GB and makes no call after it."""
    import torch
    a, b = gpu.Context(0), gpu.Context(0)
    _oracle(b, 1).close()  # the kernels are loaded before memory gets short
    b.synchronize()
    o = _oracle(a, 9)
    fill = torch.empty(_free() - (700 << 20), dtype=torch.uint8, device="cuda")
    o.close()
    assert torch.cuda.mem_get_info()[0] < 800 << 20  # the context keeps it
    if who == "context":
        _oracle(b, 10).close()  # 1 GB of tables
    else:
        del_me = torch.empty(960 << 20, dtype=torch.uint8, device="cuda")
        del del_me
    del fill
    torch.cuda.empty_cache()
    a.close()
    b.close()
