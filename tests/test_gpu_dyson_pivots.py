"""GPU check of the LU Dyson solve with tiny pivots: systems whose every step is exact in double precision.

One k point, two orbitals, V^0 = diag(1, 0), V^1 = diag(e, 1) and G = -1 for all tau give P0 = -2 [[1, e], [e, 1 + e^2]];
with one transform element -1/2, P~ = [[1, e], [e, 1]] and I - P~ = -[[0, e], [e, 0]], so W~ = -[[1, 1/e], [1/e, 1]]: with e a
power of two no operation rounds, and the pivots are e."""
import numpy as np
import pytest

from green_gpu_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [40, 300, 530])
def test_tiny_pivots(power):
    e = 2.0 ** -power
    T = 4
    V = np.zeros((1, 2, 2, 2), np.complex128)
    V[0, 0] = np.diag([1.0, 0.0])
    V[0, 1] = np.diag([e, 1.0])
    G = np.zeros((T, 1, 1, 2, 2), np.complex128)
    G[:] = -np.eye(2)
    ctx = native.Context(1, 1, 1, 2, 2, 1, T, 1)
    try:
        z, o = np.zeros(1, np.int64), np.zeros((1, 1), np.int64)
        ctx.set_symmetry(z, z, z, z, z, z, o, o)
        ctx.set_kpairs(1, z, z, z)
        ctx.set_coulomb(V)
        ctx.set_ir(np.ones((T, 1), np.complex128), np.array([[-0.5, 0.0]], np.complex128))
        _, cap = ctx.gw_sigma(G, solver=native.SOLVER_LU, capture=True)
    finally:
        ctx.close()
    assert np.array_equal(cap["Pw"][0, 0], np.array([[1.0, e], [e, 1.0]]))
    W = -np.array([[1.0, 1.0 / e], [1.0 / e, 1.0]])
    assert np.array_equal(cap["Wt"][0], np.broadcast_to(W, (T, 2, 2)))
