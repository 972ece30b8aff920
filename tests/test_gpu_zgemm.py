"""GPU check of the FP64 GEMM's tile shapes and split reductions at their edges.

Sizes sit on, below and above tile edges (8, 16, 32, 56, 64, 80), around the reduction's group of 4
and pair of groups, and where the choice of shape and split-K factor changes.  Componentwise bound: a
complex dot product of length K is two real ones of length 2K, so with u = 2^-53
|C - A B| <= sqrt(2) (2K + s) u |A||B| for any summation order (s <= 512 partial sums), and the
reference's own error has the same bound."""
import numpy as np
import pytest

from green_gpu_b200 import native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(2, 2, 2, 2, 4, 1, 4, 3)
    yield c
    c.close()


@pytest.mark.parametrize("M,N,K", [
    (1, 1, 1), (7, 9, 3), (8, 8, 4), (16, 17, 5), (33, 31, 8), (52, 52, 52), (65, 56, 12),   # one or few tiles
    (192, 195, 8), (192, 200, 384), (190, 198, 387), (9, 1, 383),                              # small kernel and its limits
    (2000, 7, 9), (1999, 20, 20), (3000, 26, 26), (2050, 37, 41), (4000, 45, 13), (5000, 52, 52),  # one column tile
    (640, 400, 33), (700, 161, 100), (513, 321, 7), (2704, 400, 30),                          # wide tiles
    (64, 64, 4099), (52, 30, 9001), (403, 611, 2707), (9, 700, 1201),                          # split reductions
    (20, 20, 33333), (36, 36, 40000), (48, 47, 9999), (55, 56, 25001)])                        # hundreds of partial sums
def test_fp64_zgemm_tile_edges(ctx, M, N, K):
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A = rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))
    B = rng.standard_normal((K, N)) + 1j * rng.standard_normal((K, N))
    out = ctx.zgemm(A, B)
    bound = 2.0 * np.sqrt(2.0) * (2 * K + 512) * 2.0 ** -53 * (np.abs(A) @ np.abs(B))
    assert (np.abs(out - A @ B) <= bound).all()
    assert np.array_equal(out, ctx.zgemm(A, B))  # a fixed summation order
