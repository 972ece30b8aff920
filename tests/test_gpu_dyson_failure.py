"""GPU check that a failing Dyson solve ends an eager build soon after it, not after the whole Sigma phase, and leaves the
context usable: launches of the failing build against those of one that succeeds."""
import numpy as np
import pytest

from green_gpu_b200 import native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [native.PREC_FP64, native.PREC_SPLIT])
def test_failure_ends_the_build(precision):
    s = synth.make_system(mesh=(2, 2, 2), nao=4, NQ=40, ns=1, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=3)
    s.V_stored = 6.0 * s.V_stored * np.exp(0.1 * np.arange(40))[None, :, None, None]
    ctx = native.context_for(s)
    try:
        good = 0.1 * s.V_stored
        ctx.set_coulomb(good)
        ref = ctx.gw_sigma(s.G_tskij, precision=precision)
        whole = ctx.launch_count()
        ctx.set_coulomb(s.V_stored)
        ctx.set_ir(s.Ttn_FB, -s.Tnt_BF)  # I - P~ indefinite
        with pytest.raises(native.GreenError) as e:
            ctx.gw_sigma(s.G_tskij, precision=precision)
        assert e.value.code == native.GG_ERR_NOT_HPD and "q_ibz" in str(e.value)
        assert ctx.launch_count() < 0.6 * whole
        ctx.set_coulomb(good)
        ctx.set_ir(s.Ttn_FB, s.Tnt_BF)
        assert np.array_equal(ctx.gw_sigma(s.G_tskij, precision=precision), ref)
    finally:
        ctx.close()
