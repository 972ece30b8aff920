"""GPU check of the FP64 products W~^T V, whose rows (tau, Q) of several tau share
tiles of 64: auxiliary sizes that fill a tile alone, with other tau, never, and more than one tile per tau;
time-reversal partners (conjugated W~) and spins.  Tolerance: the repository's parity tolerance against
the FP64 oracle, 1e-10."""
import numpy as np
import pytest

from green_gpu_b200 import native, synth
from oracle import gw as ogw

pytestmark = pytest.mark.gpu

TOL = 1e-10


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("NQ,ns", [(1, 1), (16, 2), (21, 1), (63, 1), (64, 1), (72, 2), (100, 1)])
def test_grouped_tau_rows(NQ, ns):
    s = synth.make_system(mesh=(3, 1, 1), nao=3, NQ=NQ, ns=ns, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=NQ,
                          symmetry="tr")
    ctx = native.context_for(s)
    try:
        out = ctx.gw_sigma(s.G_tskij, solver=native.SOLVER_LU)
    finally:
        ctx.close()
    assert rel(out, ogw.gw_build(s, solver="lu")) < TOL
