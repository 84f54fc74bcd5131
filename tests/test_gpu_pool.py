"""The context's device-memory pool: what it keeps when idle is bounded, it is
given back when the context ends, and contexts of several threads allocate and
free side by side with the right results."""
import threading

import numpy as np
import pytest

import oracle as O
from nightstream_b200 import gpu

pytestmark = pytest.mark.gpu
KEEP = 1 << 30


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_pool_is_bounded_and_given_back():
    slack = 256 << 20  # the context's own buffers and the driver's
    before = _free()
    c = gpu.Context(0)
    o = gpu.GpuMemOracle(c, gpu.MEM_PRODUCT, np.zeros((20, 1 << 22, 2), np.uint64))  # 1.3 GB of columns, 2 GB in all
    assert _free() < before - KEEP
    o.close()
    c.synchronize()
    assert _free() >= before - KEEP - slack
    c.close()
    assert _free() >= before - slack


def test_threads_with_their_own_contexts():
    errors = []

    def work(seed):
        try:
            rng = np.random.default_rng(seed)
            c = gpu.Context(0)
            for m in (1000, 70000, 333):
                z = rng.integers(0, 1 << 40, size=m, dtype=np.uint64)
                Z = c.decomp_b2(z)
                if not np.array_equal(Z, O.decomp_b2(z)):
                    raise AssertionError(f"decomp {m}")
                mix = c.rlc_mix(rng.integers(-2, 3, size=(2, 54)), np.stack([Z, Z]))
                planes, _ = c.split_b(mix)
                if not np.array_equal((planes.astype(np.int64) << np.arange(12).reshape(12, 1, 1)).sum(0), mix):
                    raise AssertionError(f"split {m}")
            c.close()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    ts = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
