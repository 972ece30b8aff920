"""The GW planner's chunks against the buffers that a build allocates."""
import ctypes

import pytest

import internals
from green_gpu_b200 import native


def plan(shape, solver, budget, slices=0):
    out = (ctypes.c_int64 * 5)()
    s = native.Shape(*shape, 0)
    rc = internals.load().plan_work(ctypes.byref(s), s.ns, slices, solver, ctypes.c_int64(budget), out)
    return rc, dict(zip(("qc", "kc", "tb", "dys", "bytes"), out))


def buffers(shape, solver, p):
    """Bytes of the work buffers of a build with plan p (FP64)."""
    nk, ink, nq, inq, n, N, ns, T, nw = shape
    T2, nn, NN = T // 2, n * n, N * N
    b = 2 * nk * ns * T * nn + p["kc"] * (N + T2) * nn
    b += 2 * max(p["kc"] * p["tb"] * N * nn, T * max(N * nn, NN))
    b += p["qc"] * (T2 + nw + T) * NN + T * NN + (1 << 22)
    dys = min(p["dys"], p["qc"] * nw)
    b += dys * NN
    if solver == native.SOLVER_LU:
        lub = 32 if (N | 1) * 32 * 16 <= 220 * 1024 else 16
        b += dys * -(-N // lub) * lub * lub
    return 16 * b


@pytest.mark.parametrize("solver", [native.SOLVER_CHOLESKY, native.SOLVER_LU])
@pytest.mark.parametrize("shape", [(64, 64, 64, 64, 52, 400, 1, 72, 69), (8, 8, 8, 8, 26, 120, 2, 72, 69),
                                   (1, 1, 1, 1, 20, 140, 1, 24, 21), (4, 4, 4, 4, 3, 450, 1, 24, 21),
                                   (1, 1, 1, 1, 1, 1000, 1, 4, 1)])
def test_chunks_fit_the_budget(shape, solver):
    rc, full = plan(shape, solver, 1 << 50)
    assert rc == native.GG_OK and full["qc"] == shape[3] and full["kc"] == shape[0]
    assert full["bytes"] == buffers(shape, solver, full)
    # the smallest work space that builds without the inverses of LU's diagonal blocks were accepted with
    nk, ink, nq, inq, n, N, ns, T, nw = shape
    least = buffers(shape, native.SOLVER_CHOLESKY, dict(qc=1, kc=1, tb=1, dys=592))
    for frac in (1.0, 0.7, 0.4, 0.2, 0.1, 0.03):
        budget = int(full["bytes"] * frac)
        rc, p = plan(shape, solver, budget)
        if budget < least and rc != native.GG_OK:
            assert rc == native.GG_ERR_MEMORY
            continue
        assert rc == native.GG_OK
        assert p["bytes"] == buffers(shape, solver, p)
        assert p["bytes"] <= budget or buffers(shape, native.SOLVER_CHOLESKY, p) <= budget and p["dys"] == 1
    assert plan(shape, solver, least)[0] == native.GG_OK
