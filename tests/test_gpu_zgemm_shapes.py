"""GPU check of every tile shape of the FP64 GEMM in every operand layout, through the internal descriptor: tile edges,
reductions over K-batches, split reductions, two-level index maps, three-level batches, conjugation, alpha and beta, the
three-product form, products in place and lower triangles.

Bounds: a complex dot product of length L = KB K is two real ones of length 2 L, so for any summation order
|C - ref| <= 2 sqrt(2) (2 L + s + 8) u (|alpha| |A||B| + |beta| |C0|) componentwise (s partial sums, the reference's own
error included).  With three products the bound holds with |x| = |re| + |im| and a factor of 3 (three products, sums
of their operands)."""
import ctypes

import numpy as np
import pytest

import internals

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LAYOUTS = ["kk", "kn", "nk", "nn"]


class Product:
    """C[b] = alpha sum_kb op(A[b, kb]) op(B[b, kb]) + beta C[b] on the GPU and in numpy."""

    def __init__(self, layout, M, N, K, KB=1, batch=(1, 1, 1), conj=(0, 0), gauss=0, split_rows=0, seed=0):
        rng = np.random.default_rng(seed)
        z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
        nb0, nb1, nb2 = batch
        self.shape, self.gauss, self.split_rows = (M, N, K, KB), gauss, split_rows
        self.batch, self.conj, self.layout = batch, conj, layout
        # batch levels slowest first; A does not depend on the middle level
        self.A = z(nb2, nb0, KB, M, K)
        self.B = z(nb2, nb1, nb0, KB, K, N)
        self.C0 = z(nb2, nb1, nb0, M, N)

    def _opA(self):
        return np.conj(self.A) if self.conj[0] else self.A

    def _opB(self):
        return np.conj(self.B) if self.conj[1] else self.B

    def ref(self, alpha, beta):
        size = (lambda x: np.abs(x.real) + np.abs(x.imag)) if self.gauss else np.abs
        out = (self._opA()[:, None] @ self._opB()).sum(axis=3)
        mag = (size(self.A)[:, None] @ size(self.B)).sum(axis=3)
        return alpha * out + beta * self.C0, abs(alpha) * mag + abs(beta) * np.abs(self.C0)

    def run(self, shape, splits=1, alpha=1.0, beta=0.0, inplace=0, tri=None):
        import torch
        M, N, K, KB = self.shape
        nb0, nb1, nb2 = self.batch
        up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
        A = up(self.A if self.layout[0] == "k" else np.swapaxes(self.A, -1, -2))
        B = up(np.swapaxes(self.B, -1, -2) if self.layout[1] == "k" else self.B)
        a_m, a_k = ((0, 0, K), 1) if self.layout[0] == "k" else ((0, 0, 1), M)
        b_n, b_k = ((0, 0, K), 1) if self.layout[1] == "k" else ((0, 0, 1), N)
        s, C0 = self.split_rows, self.C0
        if s:  # C in column blocks of s: [n / s][m][n % s], its rows in two levels as well
            c_m, c_n = (s, s * s, s), (s, s * M, 1)
            C0 = np.swapaxes(C0.reshape(*C0.shape[:-1], N // s, s), -2, -3)
        else:
            c_m, c_n = (0, 0, N), (0, 0, 1)
        C = up(C0)
        a_b = (KB * M * K, 0, nb0 * KB * M * K)
        b_b = (KB * K * N, nb0 * KB * K * N, nb1 * nb0 * KB * K * N)
        c_b = (M * N, nb0 * M * N, nb1 * nb0 * M * N)
        if inplace == 1:
            C = A
        elif inplace == 2:
            C = B
        total = nb0 * nb1 * nb2 * M * N
        work = torch.empty(total * splits, dtype=torch.complex128, device="cuda") if splits > 1 else None
        flag = None if tri is None else torch.tensor([tri], dtype=torch.int32, device="cuda")
        v = [M, N, K, KB, *a_m, a_k, M * K, *b_n, b_k, K * N, *c_m, *c_n, nb0, nb1, nb2, *a_b, *b_b, *c_b, *self.conj,
             self.gauss, inplace, 0 if work is None else work.numel()]
        alpha, beta = complex(alpha), complex(beta)
        torch.cuda.synchronize()
        p = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)
        n = internals.load().zgemm_desc((ctypes.c_int64 * len(v))(*v), (ctypes.c_double * 4)(alpha.real, alpha.imag, beta.real, beta.imag),
                                        p(A), p(B), p(C), p(work), p(flag), shape, splits)
        assert n > 0
        out = C.cpu().numpy().reshape(C0.shape)
        return np.swapaxes(out, -2, -3).reshape(self.C0.shape) if s else out

    def check(self, shape, splits=1, alpha=1.0, beta=0.0, inplace=0, tri=None):
        out = self.run(shape, splits, alpha, beta, inplace, tri)
        ref, mag = self.ref(alpha, beta)
        L = self.shape[2] * self.shape[3]
        bound = 2.0 * np.sqrt(2.0) * (3 if self.gauss else 1) * (2 * L + splits + 8) * U * mag
        ok = np.abs(out - ref) <= bound
        if tri:
            ok = np.tril(ok) | ~np.tril(np.ones(ok.shape[-2:], bool))
        assert ok.all(), (self.layout, self.shape, shape, splits, inplace, tri)


def tiles(gauss):
    lib = internals.load()
    t = (ctypes.c_int64 * 3)()
    out = []
    for i in range(lib.zgemm_shapes(gauss)):
        lib.zgemm_tile(gauss, i, t)
        out.append((i, t[0], t[1], t[2]))
    return out


@pytest.mark.parametrize("layout,gauss", [(l, 0) for l in LAYOUTS] + [("kk", 1), ("kn", 1)])
def test_every_shape(layout, gauss):
    for i, bm, bn, teams in tiles(gauss):
        Product(layout, bm, bn, 8, seed=i, gauss=gauss).check(i)                                # one whole tile
        Product(layout, 1, 1, 1, seed=i, gauss=gauss).check(i)
        Product(layout, bm + 1, 2 * bn - 1, 13, KB=3, conj=(1, 0), seed=i, gauss=gauss).check(i, alpha=0.5 - 2j, beta=1.5j)
        Product(layout, 2 * bm + 7, bn - 1, 30, batch=(2, 3, 2), conj=(0, 1), seed=i, gauss=gauss).check(i)
        Product(layout, bm - 1, bn + 3, 5, KB=17, batch=(3, 1, 1), seed=i, gauss=gauss).check(i, splits=4, alpha=-1.0, beta=1.0)
        Product(layout, 3 * bm, 2 * bn, 7, KB=40, seed=i, gauss=gauss).check(i, splits=37)        # two-level sum of the parts
        Product(layout, 36, 24, 9, batch=(1, 2, 1), conj=(1, 1), split_rows=12, seed=i, gauss=gauss).check(i, beta=-1.0)


@pytest.mark.parametrize("gauss", [0, 1])
def test_many_tiles_per_team(gauss):
    # more tiles than go out as a CTA each: persistent CTAs, second teams, the staggered start
    for i, bm, bn, teams in tiles(gauss):
        n = 148 * 4 * teams + 5
        Product("kn", bm, bn - 1, 6, batch=(n // 3 + 1, 3, 1), seed=i, gauss=gauss).check(i)


@pytest.mark.parametrize("layout", ["kk", "kn"])
def test_in_place(layout):
    for i, bm, bn, teams in tiles(0):
        if bn >= 24:
            p = Product(layout, 3 * bm + 5, bn - 3, bn - 3, batch=(2, 1, 1), seed=i)  # C overlays A: same rows, N = K
            p.check(i, inplace=1)
        if bm >= 32 and layout == "kn":
            p = Product(layout, bm - 1, 2 * bn + 3, bm - 1, batch=(2, 1, 1), seed=i)  # C overlays B: same columns, M = K
            p.check(i, inplace=2)


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("flag", [0, 1])
def test_lower_triangle(layout, flag):
    for i, bm, bn, teams in tiles(0):
        for n, splits in ((bn, 1), (2 * bm + 1, 3), (150, 1)):
            Product(layout, n, n, 40, batch=(2, 1, 1), seed=i).check(i, splits=splits, tri=flag)


@pytest.mark.parametrize("layout", LAYOUTS)
def test_small_kernel_and_choice(layout):
    for M, N, K, KB in ((1, 1, 1, 1), (9, 17, 3, 2), (52, 52, 52, 1), (64, 72, 5, 19), (100, 100, 100, 1), (300, 40, 7, 11)):
        Product(layout, M, N, K, KB=KB, batch=(2, 1, 2), conj=(1, 0), seed=M).check(-1, alpha=2.0 + 1j, beta=0.5)
