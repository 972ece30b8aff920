"""GPU check of the LU Dyson solve where the panel no longer fits shared memory (16 columns of N > 879 rows) and is
factored in place in global memory, against numpy: positive definite systems and indefinite ones, whose rows are
really interchanged.

Bound as for any backward stable solve: c N u cond(A) ||W||, plus nw u of the transforms' sums."""
import numpy as np
import pytest

from green_gpu_b200 import native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NQ,sign", [(879, 1), (880, 1), (880, -1), (897, -1)])
def test_lu_panel_in_place(NQ, sign):
    s = synth.make_system(mesh=(1, 1, 1), nao=3, NQ=NQ, ns=1, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=NQ,
                          with_V=False)
    rng = np.random.default_rng(NQ)
    V = rng.standard_normal((1, NQ, 3, 3)) + 1j * rng.standard_normal((1, NQ, 3, 3))
    V = 0.5 * (V + np.conj(np.swapaxes(V, -1, -2)))
    s.V_stored = (0.03 if sign > 0 else 0.6) * V
    s.Tnt_BF = sign * s.Tnt_BF
    ctx = native.context_for(s)
    try:
        _, cap = ctx.gw_sigma(s.G_tskij, solver=native.SOLVER_LU, capture=True)
    finally:
        ctx.close()
    P = cap["Pw"][0]
    A = np.eye(NQ) - P
    e = np.linalg.eigvalsh(A)
    assert e.min() > 0 if sign > 0 else e.min() < 0
    W = np.linalg.solve(A, P)
    W = 0.5 * (W + np.conj(np.swapaxes(W, 1, 2)))
    ref = np.tensordot(s.Ttn_FB, W, axes=(1, 0))
    cond = (np.abs(e).max(axis=1) / np.abs(e).min(axis=1)).max()
    scale = np.abs(s.Ttn_FB).sum(axis=1).max() * np.abs((1.0 - e) / e).max()  # W = A^-1 - I
    assert np.abs(cap["Wt"][0] - ref).max() <= 16 * (NQ + 21) * 2.0 ** -53 * cond * scale
