"""Fold steps whose chunk has no Twist access (the address-lane claims have no items) or no
access of any kind, proof words and transcript bit for bit against the oracle."""
import numpy as np
import pytest

from nightstream_b200 import gpu, synth
from oracle.fold import OracleShard

pytestmark = pytest.mark.gpu
Q = (1 << 64) - (1 << 32) + 1


@pytest.mark.parametrize("lookup_rate", [1.0, 0.0])
def test_steps_without_twist_events(ctx, lookup_rate):
    ell = 10
    ccs, z, mem = synth.make_memory_workload(ell, 5, 16, 6, 5, rw_rate=0.0, lookup_rate=lookup_rate)
    pp = np.random.default_rng(ell + 5).integers(0, Q, size=(16, 1 << ell, 54), dtype=np.uint64)
    ctx.pp_upload(pp)
    g = gpu.Shard(ctx, ccs, m_in=1, k_rho=12, app_label=b"neo/test-idle", mem=mem)
    o = OracleShard(ccs, pp, m_in=1, k_rho=12, app_label=b"neo/test-idle", mem=mem)
    for s in range(2):
        pg, po = g.fold_step(z), o.fold_step(z)
        assert np.array_equal(pg, po), f"step {s}: first mismatch at word {int(np.argmax(pg != po))}"
        assert np.array_equal(g.transcript_state(), o.tr.state()), f"step {s}"
    g.close()
