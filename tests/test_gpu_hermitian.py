"""GPU check of the lower-triangle polarisation of FP64 builds: with Hermitian G(tau) P0 is Hermitian and only its
tiles on and below the diagonal are computed, any other G takes all of them; the device decides for each
call.

Which path ran is visible in the captured P0: the short one mirrors, so P0 equals its adjoint bit for
bit.  Tolerance: the repository's parity tolerance against the FP64 oracle, 1e-10; auxiliary sizes around
the tile edges, both spins, spinors."""
import numpy as np
import pytest

from green_gpu_b200 import native, synth
from oracle import gw as ogw

pytestmark = pytest.mark.gpu

TOL = 1e-10


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def adjoint(x):
    return np.conj(np.swapaxes(x, -1, -2))


def build(s, x2c=False, graph=False):
    ctx = native.context_for(s)
    try:
        if x2c:
            ctx.set_x2c(True)
        out, cap = ctx.gw_sigma(s.G_tskij, capture=True)
        if graph:
            ctx.set_graph(True)
            ctx.gw_sigma(s.G_tskij)
            out = ctx.gw_sigma(s.G_tskij)
    finally:
        ctx.close()
    return out, cap["P0"]


@pytest.mark.parametrize("nao,NQ,ns,symm", [(3, 1, 1, "none"), (4, 17, 2, "tr"), (6, 41, 1, "tr"), (5, 64, 1, "none"),
                                            (5, 81, 2, "none"), (8, 130, 1, "tr"), (3, 257, 1, "none")])
def test_hermitian_and_general_g(nao, NQ, ns, symm):
    s = synth.make_system(mesh=(2, 1, 1), nao=nao, NQ=NQ, ns=ns, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=NQ,
                          symmetry=symm)
    out, P0 = build(s)
    assert np.array_equal(P0, adjoint(P0))
    assert rel(out, ogw.gw_build(s)) < TOL
    # a general G, far from Hermitian and by a hair
    rng = np.random.default_rng(nao)
    noise = rng.standard_normal(s.G_tskij.shape) + 1j * rng.standard_normal(s.G_tskij.shape)
    hermitian = s.G_tskij
    for size in (0.05, 1e-11):
        s.G_tskij = hermitian * (1.0 + size * noise)
        general, P0 = build(s)
        if NQ > 1:
            assert not np.array_equal(P0, adjoint(P0))
        assert rel(general, ogw.gw_build(s)) < TOL
    assert rel(general, out) < 1e-9


def test_one_matrix_that_is_not_hermitian_is_enough():
    s = synth.make_system(mesh=(2, 1, 1), nao=5, NQ=70, ns=2, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=2)
    s.G_tskij[7, 1, 1, 3, 0] += 0.03j
    out, P0 = build(s, graph=True)
    assert not np.array_equal(P0, adjoint(P0))
    assert rel(out, ogw.gw_build(s)) < 1e-10


def test_spinor_blocks_pair_up():
    s = synth.make_x2c_system(mesh=(2, 1, 1), nao=4, NQ=70, seed=4)
    _, P0 = build(s, x2c=True)
    assert np.array_equal(P0, adjoint(P0))
    s.G_tskij[3, 0, 0, 1, 6] *= 1.01  # ab no longer the adjoint of ba
    _, P0 = build(s, x2c=True)
    assert not np.array_equal(P0, adjoint(P0))
