"""GPU check of FP64 builds whose G(tau) is Hermitian only to rounding, within the limit up to which the lower triangle
of P0 is computed and mirrored.

The Hermitian part of P0, which is all that the Dyson step uses, depends on the anti-Hermitian part of G in second
order only: 2^-92 at the limit, nothing in double precision.  So P~ must be the same, bit for bit, for G and for
its Hermitian part."""
import ctypes

import numpy as np
import pytest

from green_gpu_b200 import native, synth

pytestmark = pytest.mark.gpu


def p_tilde(s, G, x2c):
    ctx = native.context_for(s)
    try:
        if x2c:
            ctx.set_x2c(True)
        P = np.empty((s.inq, s.nw_b, s.NQ, s.NQ), np.complex128)
        ctx._check(ctx.lib.gg_set_capture(ctx.h, None, P.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None))
        ctx.gw_sigma(G, solver=native.SOLVER_LU)
    finally:
        ctx.close()
    return P


@pytest.mark.parametrize("nao,NQ,ns,symm,x2c", [(8, 48, 1, "tr", False), (33, 70, 2, "none", False),
                                                (5, 130, 1, "none", False), (6, 33, 1, "none", True)])
def test_rounding_sized_anti_hermitian_part_drops_out(nao, NQ, ns, symm, x2c):
    if x2c:
        s = synth.make_x2c_system(mesh=(2, 1, 1), nao=nao, NQ=NQ, seed=NQ)
    else:
        s = synth.make_system(mesh=(2, 1, 1), nao=nao, NQ=NQ, ns=ns, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=NQ,
                              symmetry=symm)
    rng = np.random.default_rng(nao)
    G = s.G_tskij * (1.0 + 2.0 ** -48 * rng.uniform(-1.0, 1.0, s.G_tskij.shape))
    H = 0.5 * (G + np.conj(np.swapaxes(G, -1, -2)))
    assert not np.array_equal(G, H)
    assert np.array_equal(p_tilde(s, G, x2c), p_tilde(s, H, x2c))


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("at", [(7, 0, 0, 3, 0), (7, 0, 1, 2, 2)])
def test_nan_or_infinity_in_one_component_is_not_hermitian(value, at):
    # one tau of P0 is lost either way; the others show that the whole product was computed, not its lower triangle
    s = synth.make_system(mesh=(2, 1, 1), nao=5, NQ=70, ns=1, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=2)
    G = s.G_tskij.copy()
    G.imag[at] = value
    P0 = np.empty((s.inq, s.nts, s.NQ, s.NQ), np.complex128)
    ctx = native.context_for(s)
    try:
        ctx._check(ctx.lib.gg_set_capture(ctx.h, P0.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None, None))
        with pytest.raises(native.GreenError) as e:
            ctx.gw_sigma(G, solver=native.SOLVER_LU)
        assert e.value.code == native.GG_ERR_SINGULAR
    finally:
        ctx.close()
    assert not np.isfinite(P0[:, 7]).any()
    rest = P0[:, [t for t in range(12) if t != 7]]
    assert np.isfinite(rest).all()
    assert not np.array_equal(rest, np.conj(np.swapaxes(rest, -1, -2)))
