"""An oracle's creation does the same work whatever was created before it: nothing is kept from
one call for the next."""
import numpy as np
import pytest

from memcase import rand_k
from nightstream_b200 import gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n_cols", [(gpu.MEM_SHOUT_VALUE, 2), (gpu.MEM_BITNESS, 5)])
def test_second_oracle_of_a_point_launches_as_much(ctx, kind, n_cols):
    rng = np.random.default_rng(kind)
    point, w = rand_k(rng, 8), rand_k(rng, n_cols)
    launches, claims = [], []
    cols = rand_k(rng, n_cols << 8).reshape(n_cols, 256, 2)
    for _ in range(2):
        before = ctx.kernel_launches
        o = gpu.GpuMemOracle(ctx, kind, cols, point, None, None, w)
        launches.append(ctx.kernel_launches - before)
        claims.append(o.claim.copy())
        o.close()
    assert launches[0] == launches[1]
    assert np.array_equal(*claims)
