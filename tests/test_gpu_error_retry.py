"""A call that reported a device wait that ran out leaves nothing behind: the same call again
forms its results anew, and calls that had no part in it do not see the error."""
import numpy as np
import pytest

import oracle as O
from helpers import D_SC, ELL_D, XS, ccs_case
from nightstream_b200 import gpu

pytestmark = pytest.mark.gpu


def _after_row_rounds(ctx, ell, k):
    ccs, _, Z, ch, chals = ccs_case(ell, k, True)
    args = (ccs, Z, 2, ch["alpha"], ch["beta_a"], ch["beta_r"], ch["gamma"], ch["r_inputs"], ELL_D, ell, D_SC)
    g, o = gpu.GpuCcsOracle(ctx, *args), O.CcsOracle(*args)
    for r in chals[:ell]:
        g.evals_at(XS)
        o.evals_at(XS)
        g.fold(r)
        o.fold(r)
    return g, o


@pytest.mark.parametrize("call", ["me_outputs", "evals_at"])
def test_me_outputs_are_formed_again_after_an_error(ctx, call):
    g, o = _after_row_rounds(ctx, 6, 3)
    run = (lambda x: x.me_outputs()) if call == "me_outputs" else (lambda x: (x.evals_at(XS),))
    ctx.wait_probe_async(2000)  # runs out while the call's launches wait behind it
    with pytest.raises(gpu.NeoGpuError) as e:
        run(g)
    assert e.value.code == 4 and "timed out" in str(e.value)
    before = ctx.kernel_launches
    again = run(g)
    assert ctx.kernel_launches >= before + 3  # transposed products, y, scalars: not the copies that failed
    for a, b in zip(again, run(o)):
        assert np.array_equal(a, b)
    g.close()


def test_one_report_clears_both_error_words(ctx):
    ctx.wait_probe_async(1000)
    with pytest.raises(gpu.NeoGpuError):
        ctx.wait_probe(False, spin_limit=1000)  # both words are set by then
    ctx.wait_probe(True)
    ctx.synchronize()
