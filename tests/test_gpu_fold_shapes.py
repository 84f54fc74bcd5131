"""Parts of a fold step at the edges of their shapes: the RLC mix, the digit split at whole and ragged
eights over its ranges, and bus openings of chunks that begin at any byte, and of
aligned ones with a short last tile."""
import numpy as np
import pytest

import oracle as O
from oracle.fold import OracleShard
from nightstream_b200 import gpu, synth

pytestmark = pytest.mark.gpu
Q = (1 << 64) - (1 << 32) + 1


@pytest.mark.parametrize("count,m", [(1, 1), (1, 128), (2, 4), (3, 101), (13, 127), (13, 129), (12, 260), (64, 1022), (5, 16383)])
def test_rlc_mix_shapes(ctx, count, m):
    """Column tiles with a remainder, rows on any byte, an odd witness out, full int8."""
    rng = np.random.default_rng(count * 1000 + m)
    rho = rng.integers(-2, 3, size=(count, 54)).astype(np.int8)
    Zs = rng.integers(-128, 128, size=(count, 54, m)).astype(np.int8)
    assert np.array_equal(ctx.rlc_mix(rho, Zs), O.rlc_mix(rho, Zs))


@pytest.mark.parametrize("n,k,b", [(8, 1, 2), (8, 12, 2), (2056, 12, 2), (4097, 12, 2), (4100, 30, 2), (4096, 31, 2),
                                   (4096, 5, 3)])
def test_split_shapes(ctx, n, k, b):
    rng = np.random.default_rng(n + k)
    top = min(b**k - 1, 2**31 - 1) if b == 2 else (b**k - 1) // 2
    mix = rng.integers(-top, top + 1, size=(1, n)).astype(np.int32)
    mix[0, :4] = [top, -top, 0, -1]
    planes, nz = ctx.split_b(mix, k, b)
    p2, nz2 = O.split_b(mix, k, b)
    assert np.array_equal(planes, p2) and np.array_equal(nz, nz2)
    zero, nz = ctx.split_b(np.zeros((1, n), np.int32), k, b)
    assert not zero.any() and not nz.any()
    if b == 2 and k < 31:
        for bad in (top + 1, -top - 1, -(2**31)):
            mix[0, n - 1] = bad
            with pytest.raises(gpu.NeoGpuError) as e:
                ctx.split_b(mix, k, b)
            assert e.value.code == 3


@pytest.mark.parametrize("ell,chunk,shout_ell,twist_ell", [(10, 17, 4, 3), (10, 16, 4, 3), (12, 48, 5, 4), (14, 515, 4, 3), (14, 528, 4, 3)])
def test_bus_openings_of_ragged_and_aligned_chunks(ctx, ell, chunk, shout_ell, twist_ell):
    ccs, z, mem = synth.make_memory_workload(ell, 5, chunk, shout_ell, twist_ell)
    pp = np.random.default_rng(ell).integers(0, Q, size=(16, 1 << ell, 54), dtype=np.uint64)
    ctx.pp_upload(pp)
    g = gpu.Shard(ctx, ccs, m_in=1, k_rho=12, app_label=b"neo/test-bus", mem=mem)
    o = OracleShard(ccs, pp, m_in=1, k_rho=12, app_label=b"neo/test-bus", mem=mem)
    pg, po = g.fold_step(z), o.fold_step(z)
    assert np.array_equal(pg, po), f"first mismatch at word {int(np.argmax(pg != po))}"
    g.close()
