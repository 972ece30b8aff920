"""GPU check of a GW build whose auxiliary basis has more pairs of 32 x 32 tiles (NQ > 11552) than a grid's second dimension.

One orbital and one k point make P~ of rank one, P~ = p v v^H, and Sigma that of the system with the single auxiliary
function |v|: the same build at NQ = 1 is the reference.  Rounding: sums of NQ terms."""
import numpy as np
import pytest

from green_gpu_b200 import native

pytestmark = pytest.mark.gpu


def sigma(v, G, Ttn, Tnt):
    T, nw = Ttn.shape
    ctx = native.Context(1, 1, 1, 1, len(v), 1, T, nw)
    try:
        z, o = np.zeros(1, np.int64), np.zeros((1, 1), np.int64)
        ctx.set_symmetry(z, z, z, z, z, z, o, o)
        ctx.set_kpairs(1, z, z, z)
        ctx.set_coulomb(v.reshape(1, len(v), 1, 1))
        ctx.set_ir(Ttn, Tnt)
        return ctx.gw_sigma(G, solver=native.SOLVER_CHOLESKY)
    finally:
        ctx.close()


def test_many_auxiliary_functions():
    NQ, T, nw = 11585, 4, 1
    rng = np.random.default_rng(1)
    v = (rng.standard_normal(NQ) / np.sqrt(NQ)).astype(np.complex128)  # real: V(k, k) is Hermitian in the orbitals
    G = -rng.uniform(0.2, 0.8, (T, 1, 1, 1, 1)).astype(np.complex128)
    Ttn = rng.uniform(0.5, 1.0, (T, nw)).astype(np.complex128)
    Tnt = rng.uniform(0.5, 1.0, (nw, T - 2)).astype(np.complex128)
    ref = sigma(np.array([np.linalg.norm(v)], np.complex128), G, Ttn, Tnt)
    out = sigma(v, G, Ttn, Tnt)
    assert np.abs(out - ref).max() <= 16 * NQ * 2.0 ** -53 * np.abs(ref).max()
