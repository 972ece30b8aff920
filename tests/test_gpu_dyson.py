"""GPU check of the blocked Dyson solve (Cholesky blocks of 64, LU panels of 32 or 16) at its edges.

A GW build returns P~ (Hermitian-symmetrised) and W~(tau); the W~(iOmega) that its captured P~ has in
numpy, taken back to tau with the same transforms, is the reference.  A = I - P~ >= I, so the solve's forward
error is at most c N u ||A|| ||W|| with a modest c; the transforms' sums of nw terms add nw u."""
import numpy as np
import pytest

from green_gpu_b200 import native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [native.SOLVER_CHOLESKY, native.SOLVER_LU])
@pytest.mark.parametrize("NQ", [1, 5, 16, 31, 32, 33, 63, 64, 65, 96, 127, 129, 200, 437, 450])
def test_dyson_block_edges(NQ, solver):
    s = synth.make_system(mesh=(1, 1, 1), nao=3, NQ=NQ, ns=1, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=NQ)
    # every row of P~ matters; small enough that the transforms' fit error leaves I - P~ positive definite
    s.V_stored = 0.2 * s.V_stored * np.exp(0.1 * np.arange(NQ))[None, :, None, None]
    ctx = native.context_for(s)
    try:
        _, cap = ctx.gw_sigma(s.G_tskij, solver=solver, capture=True)
    finally:
        ctx.close()
    P = cap["Pw"][0]
    A = np.eye(NQ) - P
    W = np.linalg.solve(A, P)
    if solver == native.SOLVER_LU:
        W = 0.5 * (W + np.conj(np.swapaxes(W, 1, 2)))
    ref = np.tensordot(s.Ttn_FB, W, axes=(1, 0))
    u = 2.0 ** -53
    cond = max(np.linalg.norm(a, 2) for a in A)
    scale = np.abs(s.Ttn_FB).sum(axis=1).max() * max(np.linalg.norm(w, 2) for w in W)
    assert np.abs(cap["Wt"][0] - ref).max() <= 16 * (NQ + 21) * u * cond * scale


def test_lu_pivots_on_indefinite_systems():
    # a complex transform makes I - P~ indefinite (Cholesky refuses it), so rows are interchanged;
    # zero integrals leave I - P~ = I and W = 0
    s = synth.make_system(mesh=(1, 1, 1), nao=4, NQ=70, ns=1, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=3)
    s.V_stored = 6.0 * s.V_stored * np.exp(0.1 * np.arange(70))[None, :, None, None]
    s.Tnt_BF = -s.Tnt_BF
    ctx = native.context_for(s)
    try:
        with pytest.raises(native.GreenError) as e:
            ctx.gw_sigma(s.G_tskij, solver=native.SOLVER_CHOLESKY)
        assert e.value.code == native.GG_ERR_NOT_HPD
        _, cap = ctx.gw_sigma(s.G_tskij, solver=native.SOLVER_LU, capture=True)
        P = cap["Pw"][0]
        A = np.eye(70) - P
        assert min(np.linalg.eigvalsh(a).min() for a in A) < 0
        W = np.linalg.solve(A, P)
        W = 0.5 * (W + np.conj(np.swapaxes(W, 1, 2)))
        ref = np.tensordot(s.Ttn_FB, W, axes=(1, 0))
        cond = max(np.linalg.cond(a) for a in A)
        scale = np.abs(s.Ttn_FB).sum(axis=1).max() * max(np.linalg.norm(w, 2) for w in W)
        assert np.abs(cap["Wt"][0] - ref).max() <= 16 * (70 + 21) * 2.0 ** -53 * cond * scale
        ctx.set_coulomb(0.0 * s.V_stored)
        assert not ctx.gw_sigma(s.G_tskij, solver=native.SOLVER_LU).any()
    finally:
        ctx.close()
