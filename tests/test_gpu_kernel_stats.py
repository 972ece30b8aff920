"""GPU check of the flops that gg_kernel_stats reports for P0: the lower triangle where only that is computed."""
import numpy as np
import pytest

from green_gpu_b200 import native, synth

pytestmark = pytest.mark.gpu


def test_p0_flops_follow_the_triangle():
    n, N, T2, nk, nq = 5, 70, 12, 2, 2
    s = synth.make_system(mesh=(2, 1, 1), nao=n, NQ=N, ns=1, beta=10.0, lam=100.0, nts=2 * T2, nw_b=21, seed=2)
    square = nq * T2 * (8.0 * N * N * n * n * nk + 12.0 * N * N)
    ctx = native.context_for(s)
    try:
        def flops(G, precision=native.PREC_FP64):
            ctx.gw_sigma(G, precision=precision)
            return ctx.kernel_stats(0)["flops"]
        assert np.isclose(flops(s.G_tskij), square * (N + 1) / (2 * N), rtol=1e-12)
        general = s.G_tskij.copy()
        general[3, 0, 0, 1, 2] *= 1.001
        assert np.isclose(flops(general), square, rtol=1e-12)
        assert np.isclose(flops(s.G_tskij, native.PREC_SPLIT), square, rtol=1e-12)
    finally:
        ctx.close()
