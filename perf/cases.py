"""Performance cases of the HF-exchange / GW self-energy library.

``listed()`` names the cases, ``draw(rng)`` makes further ones over the same ranges,
``prepare(case, seed)`` sets up what a caller holds before a call (contexts with integrals, IR
transforms and symmetry tables, and the inputs of one iteration), ``run(state)`` is one call through
the public entry points, ``work(case)`` the bytes and flops that the call cannot do without, and
``exact(case, seed)`` the same outputs from plain complex128 torch operations.

Kinds of case:

* ``zgemm``  gg_zgemm_noalloc on device buffers: the library's own FP64 complex GEMM;
* ``gw``     one GW self-energy build: from host arrays (``io = host``, as the green-mbpt plugin calls
             it) or on device buffers (``io = device``, as a program that keeps G and Sigma in HBM
             does), optionally replayed as a CUDA graph (a self-consistency loop);
* ``batch``  GW builds of several uneven systems in one CUDA graph (gg_batch_run);
* ``hf``     one Fock build (exchange, Hartree and Ewald terms) from host arrays;
* ``scf``    one iteration of a self-consistent job as serve.run_job does it: Fock, then Sigma.

Integrals are complex Gaussian with the e^{-0.1 Q} decay of the benchmark's recipe, G(tau) comes
from random Hermitian Fock matrices with eigenvalues in [-2, 2] Ha.  Grids: 72 tau / 69 bosonic
frequencies at beta 100, Lambda 1e4 (the benchmark's), 24 / 21 at beta 10, Lambda 100 (the tests').
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from green_gpu_b200 import native, synth

GRIDS = {72: (100.0, 1e4, 69), 24: (10.0, 100.0, 21)}  # nts: (beta, Lambda, nw_b)
PREC = {"fp64": native.PREC_FP64, "split": native.PREC_SPLIT}
SOLVER = {"cholesky": native.SOLVER_CHOLESKY, "lu": native.SOLVER_LU}


def _gw(name=None, **kw):
    c = dict(kind="gw", mesh="2x2x1", nao=20, NQ=120, ns=1, nts=72, symmetry="none", x2c=False, precision="fp64",
             solver="cholesky", io="device", graph=False)
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one orbital block of the benchmark system: the smallest call, launch latency
        dict(name="zgemm-block", kind="zgemm", M=52, N=52, K=52),
        # a long ragged reduction into a few hundred rows and columns (P0-like, caller-owned buffers)
        dict(name="zgemm-ragged", kind="zgemm", M=403, N=611, K=2707),
        # a Gamma-point molecule through the plugin: host arrays, its default LU solver
        _gw("gw-gamma-lu", mesh="1x1x1", nao=20, NQ=140, solver="lu", io="host"),
        # the small benchmark configuration through the plugin with its defaults
        _gw("gw-small-lu", mesh="2x2x2", nao=26, NQ=120, solver="lu", io="host"),
        # the same system in a self-consistency loop on the device, split precision, graph replay
        _gw("gw-small-split", mesh="2x2x2", nao=26, NQ=120, precision="split", graph=True),
        # the benchmark's orbitals and auxiliary basis on a smaller k mesh, both precisions
        _gw("gw-52-fp64", mesh="2x2x1", nao=52, NQ=400),
        _gw("gw-52-split", mesh="2x2x2", nao=52, NQ=400, precision="split", graph=True),
        # odd sizes, two spins, time-reversal-reduced mesh, default solver
        _gw("gw-odd-spin-split", mesh="3x1x1", nao=37, NQ=251, ns=2, symmetry="tr", precision="split", solver="lu"),
        # rotated stars (U_k, U_q) as a space group gives them
        _gw("gw-rotated-fp64", mesh="2x2x2", nao=20, NQ=160, symmetry="rot"),
        # two-component: spinor G of order 2 nao
        _gw("gw-x2c-fp64", mesh="2x1x1", nao=26, NQ=182, x2c=True),
        # uneven small systems in one graph, as a screening run over many structures batches them
        dict(name="batch-split", kind="batch", systems="2x2x1:20:140 2x1x1:36:252 1x1x1:52:312 2x2x1:26:120", nts=72,
             symmetry="tr", precision="split", solver="cholesky"),
        # the static part of an iteration on a 3x3x3 mesh
        dict(name="fock-3x3x3", kind="hf", mesh="3x3x3", nao=36, NQ=288, ns=1, symmetry="tr", precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    largest = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["zgemm", "gw", "gw", "gw", "gw", "batch", "hf", "scf"])
        if kind == "zgemm":
            c = dict(kind="zgemm", M=_log_int(rng, 16, 720), N=_log_int(rng, 16, 720), K=_log_int(rng, 16, 4000))
        elif kind == "batch":
            sys_ = []
            for _ in range(rng.randint(2, 5)):
                n = _log_int(rng, 12, 48)
                sys_.append("%s:%d:%d" % (rng.choice(["1x1x1", "2x1x1", "2x2x1"]), n, int(n * rng.uniform(5, 8))))
            c = dict(kind="batch", systems=" ".join(sys_), nts=72, symmetry=rng.choice(["none", "tr"]),
                     precision=rng.choice(["fp64", "split"]), solver=rng.choice(["cholesky", "lu"]))
        else:
            n = _log_int(rng, 10, 56)
            c = dict(kind=kind, mesh=rng.choice(["1x1x1", "2x1x1", "3x1x1", "2x2x1", "2x2x2", "3x2x2"]), nao=n,
                     NQ=int(n * rng.uniform(5, 8)), ns=rng.choice([1, 1, 2]), symmetry=rng.choice(["none", "tr", "rot"]),
                     precision=rng.choice(["fp64", "split"]))
            if kind == "hf":
                c["mesh"] = rng.choice(["2x2x1", "2x2x2", "3x2x2", "3x3x3"])
            else:
                c.update(nts=rng.choice([24, 72, 72]), solver=rng.choice(["cholesky", "lu"]))
            if kind == "gw":
                x2c = rng.random() < 0.15
                c.update(x2c=x2c, io=rng.choice(["host", "device", "device"]))
                c["graph"] = c["io"] == "device" and rng.random() < 0.5
                if x2c:
                    c.update(ns=1, symmetry="none", nao=max(6, n // 2))
        if _cost(c) <= largest:
            return c


# ------------------------------------------------------------------ inputs
def _mesh(case):
    return tuple(int(x) for x in case["mesh"].split("x"))


def _systems(case):
    """The systems of a batch case as gw cases."""
    out = []
    for item in case["systems"].split():
        mesh, nao, NQ = item.split(":")
        out.append(_gw(mesh=mesh, nao=int(nao), NQ=int(NQ), nts=case["nts"], symmetry=case["symmetry"],
                       precision=case["precision"], solver=case["solver"]))
    return out


def _unitary(rng, n):
    return np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]


def _inputs(case, seed):
    """(system tables, G, IR transforms as a synth.System; integrals on the GPU)."""
    nts = case.get("nts", 24)
    beta, lam, nw_b = GRIDS[nts]
    kw = dict(mesh=_mesh(case), nao=case["nao"], NQ=case["NQ"], beta=beta, lam=lam, nts=nts, nw_b=nw_b, seed=seed)
    rng = np.random.default_rng(seed + 77)
    if case.get("x2c"):
        s = synth.make_system(with_V=False, **kw)
        _spinor_green(s, rng, beta)
    else:
        sym = "tr" if case["symmetry"] == "rot" else case["symmetry"]
        s = synth.make_system(with_V=False, ns=case["ns"], symmetry=sym, **kw)
    if case.get("symmetry") == "rot":
        # a star member is its representative seen through a unitary rotation of the orbitals and
        # of the auxiliary basis, then conjugated
        s.U_k = np.stack([np.eye(s.nao) if s.k_reduced_to_full[s.k_full_to_reduced[k]] == k else _unitary(rng, s.nao)
                          for k in range(s.nk)]).astype(np.complex128)
        s.U_q = np.stack([np.eye(s.NQ) if s.q_reduced_to_full[s.q_full_to_reduced[q]] == q else _unitary(rng, s.NQ)
                          for q in range(s.nq)]).astype(np.complex128)
    npairs = int(s.irre_pos_kpair.max()) + 1
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    V = torch.randn((npairs, s.NQ, s.nao, s.nao, 2), dtype=torch.float64, device="cuda", generator=g)
    V = torch.view_as_complex(V)
    scale = torch.exp(-0.1 * torch.arange(s.NQ, device="cuda", dtype=torch.float64)) / math.sqrt(2.0)
    V *= scale[None, :, None, None]
    for k in range(s.nk):  # V(k, k) is Hermitian in the orbitals
        p = int(s.irre_pos_kpair[k * (k + 1) // 2 + k])
        if p >= 0:
            V[p] = 0.5 * (V[p] + V[p].mH)
    return s, V


def _spinor_green(s, rng, beta):
    """G(tau) of spinor Fock matrices of order 2 nao with coupled spin blocks."""
    n2 = 2 * s.nao
    G = np.empty((s.nts, 1, s.ink, n2, n2), np.complex128)
    t = s.tau[:, None]
    for k in range(s.ink):
        U = _unitary(rng, n2)
        e = rng.uniform(-2.0, 2.0, n2)[None, :]
        g = np.where(e >= 0, np.exp(-t * np.abs(e)), np.exp((t - beta) * np.abs(e))) / (1.0 + np.exp(-beta * np.abs(e)))
        G[:, 0, k] = -np.einsum("ia,ta,ja->tij", U, g, U.conj())
    s.G_tskij = G


def _context(case, s, V):
    ctx = native.Context(s.nk, s.ink, s.inq, s.nao, s.NQ, s.ns, s.nts, s.nw_b)
    ctx.set_symmetry(s.k_full_to_reduced, s.k_reduced_to_full, s.k_tr_conj, s.q_full_to_reduced, s.q_reduced_to_full,
                     s.q_tr_conj, s.k1_from_k2q, s.k2_from_k1q, s.U_k, s.U_q)
    ctx.set_kpairs(V.shape[0], s.conj_kpair_list, s.trans_kpair_list, s.irre_pos_kpair)
    ctx.set_coulomb_device(V.data_ptr(), keepalive=V)
    ctx.set_ir(s.Ttn_FB, s.Tnt_BF)
    if case.get("x2c"):
        ctx.set_x2c(True)
    return ctx


# ------------------------------------------------------------------ the cases
def prepare(case, seed):
    kind = case["kind"]
    if kind == "zgemm":
        A, B = _zgemm_inputs(case, seed)
        return dict(case=case, lib=native.load(), A=A, B=B, C=torch.empty((case["M"], case["N"]), dtype=A.dtype, device="cuda"))
    if kind == "batch":
        items, keep = [], []
        for i, c in enumerate(_systems(case)):
            s, V = _inputs(c, 100 * seed + i)
            G = torch.from_numpy(s.G_tskij).cuda()
            S = torch.empty_like(G)
            torch.cuda.synchronize()
            items.append((_context(c, s, V), G.data_ptr(), S.data_ptr()))
            keep.append((V, G, S))
        batch = native.Batch(items, solver=SOLVER[case["solver"]], precision=PREC[case["precision"]])
        return dict(case=case, batch=batch, keep=keep)
    s, V = _inputs(case, seed)
    torch.cuda.synchronize()
    ctx = _context(case, s, V)
    st = dict(case=case, ctx=ctx, s=s, V=V, G=s.G_tskij, dm=s.dm)
    if kind in ("hf", "scf"):
        ctx.set_hf_precision(PREC[case["precision"]])
    elif case["io"] == "device":
        st["G"] = torch.from_numpy(s.G_tskij).cuda()
        st["Sigma"] = torch.empty_like(st["G"])
        ctx.set_graph(case["graph"])
        torch.cuda.synchronize()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "zgemm":
        P = ctypes.c_void_p
        A, B, C = st["A"], st["B"], st["C"]
        rc = st["lib"].gg_zgemm_noalloc(case["M"], case["N"], case["K"], P(A.data_ptr()), P(B.data_ptr()),
                                        P(C.data_ptr()), P(torch.cuda.current_stream().cuda_stream))
        if rc != native.GG_OK:
            raise RuntimeError(st["lib"].gg_last_error(None).decode())
        return C
    if kind == "batch":
        st["batch"].run()
        return [S for _, _, S in st["keep"]]
    ctx, s = st["ctx"], st["s"]
    if kind == "hf":
        return ctx.hf_fock(st["dm"], s.S_k, s.madelung)
    solver, precision = SOLVER[case["solver"]], PREC[case["precision"]]
    if kind == "scf":
        return ctx.hf_fock(st["dm"], s.S_k, s.madelung), ctx.gw_sigma(st["G"], solver=solver, precision=precision)
    if case["io"] == "host":
        return ctx.gw_sigma(st["G"], solver=solver, precision=precision)
    ctx.gw_sigma_device(st["G"].data_ptr(), st["Sigma"].data_ptr(), solver=solver, precision=precision)
    return st["Sigma"]


def _zgemm_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    M, N, K = case["M"], case["N"], case["K"]
    A = torch.randn((M, K), dtype=torch.complex128, device="cuda", generator=g)
    B = torch.randn((K, N), dtype=torch.complex128, device="cuda", generator=g)
    return A, B


# ------------------------------------------------------------------ work
def _irreducible(case):
    """(k points, irreducible k points, stored k-pairs) of a case."""
    n1, n2, n3 = _mesh(case)
    nk = n1 * n2 * n3
    if case["symmetry"] == "none":
        return nk, nk, nk * (nk + 1) // 2
    real = 1  # k points with k = -k
    for n in (n1, n2, n3):
        real *= 2 - n % 2
    return nk, (nk + real) // 2, nk * (nk + 1) // 4 + 1


def work(case):
    """Bytes: every input read once, every output written once.  Flops: the reference's count of the
    complex GEMMs (8MNK + 12MN) and of the solver."""
    kind = case["kind"]
    if kind == "zgemm":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 16.0 * (M * K + K * N + M * N), "flops": 8.0 * M * N * K}
    if kind == "batch":
        parts = [work(c) for c in _systems(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    nk, ink, npairs = _irreducible(case)
    n, NQ = case["nao"], case["NQ"]
    ns = 4 if case.get("x2c") else case["ns"]
    b, f = 16.0 * npairs * NQ * n * n, 0.0
    if kind in ("hf", "scf"):
        b += 16.0 * 3 * ns * ink * n * n
        f += synth.hf_flop_model(nk, ink, ns, n, NQ)
    if kind in ("gw", "scf"):
        nts = case["nts"]
        b += 16.0 * 2 * nts * ns * ink * n * n
        f += synth.gw_flop_model(nk, ink, ink, ns, nts, GRIDS[nts][2], n, NQ)
    return {"bytes": b, "flops": f}


def _cost(case):
    """Rough time of a case: split precision does the contractions about three times as fast, the
    pivoted LU is a long chain of small steps."""
    f = work(case)["flops"]
    cases = _systems(case) if case["kind"] == "batch" else [case]
    chain = sum(1e-7 * c["NQ"] ** 3 * _irreducible(c)[1] * 1e12 / 20 for c in cases if c.get("solver") == "lu")
    return f / (2.0 if case.get("precision") == "split" else 1.0) + chain


# ------------------------------------------------------------------ exact results
def _pair_getter(s, V):
    """V(k1, k2) from the stored pairs: the Hermitian partner for k1 < k2, then the conjugated or
    transposed pair that the lists name."""
    def get(k1, k2):
        idx = k1 * (k1 + 1) // 2 + k2 if k1 >= k2 else k2 * (k2 + 1) // 2 + k1
        conj = trans = False
        if s.conj_kpair_list[idx] != idx:
            idx, conj = int(s.conj_kpair_list[idx]), True
        elif s.trans_kpair_list[idx] != idx:
            idx, trans = int(s.trans_kpair_list[idx]), True
        v = V[int(s.irre_pos_kpair[idx])]
        if k1 < k2:
            v = v.mH
        if conj:
            v = v.conj()
        if trans:
            v = v.mT
        return v.resolve_conj().contiguous()
    return get


def _unfolded(s, X):
    """[...][ink][n][n] -> [nk][...][n][n] through U_k and time reversal."""
    out = []
    for k in range(s.nk):
        x = X[..., int(s.k_full_to_reduced[k]), :, :]
        if s.U_k is not None:
            U = torch.from_numpy(s.U_k[k]).to(X.device)
            x = U @ x @ U.mH
        out.append(x.conj().resolve_conj() if s.k_tr_conj[k] else x)
    return torch.stack(out)


def _herm(P):
    return 0.5 * (P + P.mH)


def _exact_gw(s, V, x2c):
    dev = V.device
    G = torch.from_numpy(s.G_tskij).to(dev)
    Gf = _unfolded(s, G)  # [nk][nts][ns][n][n]
    if x2c:  # spin-independent integrals: block diagonal in the spinor space
        W = torch.zeros(V.shape[:2] + (2 * s.nao, 2 * s.nao), dtype=V.dtype, device=dev)
        W[..., :s.nao, :s.nao] = V
        W[..., s.nao:, s.nao:] = V
        V = W
    n, NQ, T, ns = G.shape[-1], s.NQ, s.nts, s.ns
    T2 = T // 2
    pair = _pair_getter(s, V)
    Ttn, Tnt = (torch.from_numpy(x).to(dev) for x in (s.Ttn_FB, s.Tnt_BF))
    pref = (-2.0 if ns == 1 and not x2c else -1.0) / s.nk
    Sigma = torch.zeros_like(G)
    eye = torch.eye(NQ, dtype=V.dtype, device=dev)
    for iq in range(s.inq):
        q = int(s.q_reduced_to_full[iq])
        P0 = torch.zeros((T, NQ, NQ), dtype=V.dtype, device=dev)
        for k in range(s.nk):
            k1 = int(s.k1_from_k2q[k * s.nq + q])
            v = pair(k, k1)
            for sp in range(ns):
                for t in range(T2):
                    a = (Gf[k, T - 1 - t, sp] @ v).reshape(NQ, n * n)
                    b = (v.conj() @ Gf[k1, t, sp].mT).reshape(NQ, n * n)
                    P0[t] += pref * (a @ b.mT)
        P0[T2:] = P0[:T2].flip(0)
        P = _herm(torch.tensordot(Tnt, P0[1:T - 1], dims=([1], [0])))
        W = torch.tensordot(Ttn, _herm(torch.linalg.solve(eye - P, P)), dims=([1], [0]))
        for qd in (int(x) for x in s.q_stars[iq]):
            Wq = W
            if s.U_q is not None:
                U = torch.from_numpy(s.U_q[qd]).to(dev)
                Wq = U @ Wq @ U.mH
            if s.q_tr_conj[qd]:
                Wq = Wq.conj().resolve_conj()
            for kr in range(s.ink):
                k1 = int(s.k2_from_k1q[int(s.k_reduced_to_full[kr]) * s.nq + qd])
                v = pair(int(s.k_reduced_to_full[kr]), k1)
                vh = v.conj().permute(0, 2, 1).reshape(NQ * n, n)
                for t in range(T):
                    x = (v.reshape(NQ, n * n).mT @ Wq[t]).reshape(n, n, NQ).permute(2, 0, 1)
                    for sp in range(ns):
                        z = (x @ Gf[k1, t, sp]).permute(1, 0, 2).reshape(n, NQ * n)
                        Sigma[t, sp, kr] -= z @ vh / s.nk
    return Sigma


def _exact_fock(s, V):
    dev = V.device
    dm = torch.from_numpy(np.ascontiguousarray(s.dm)).to(dev)
    S = torch.from_numpy(s.S_k).to(dev)
    D = _unfolded(s, dm)  # [nk][ns][n][n]
    pair = _pair_getter(s, V)
    pref = (-0.5 if s.ns == 1 else -1.0) / s.nk
    c = sum(torch.einsum("Qab,sba->Q", pair(k, k), D[k]) for k in range(s.nk)) / s.nk
    F = -(0.5 if s.ns == 1 else 1.0) * s.madelung * (S @ dm @ S)
    for kr in range(s.ink):
        k = int(s.k_reduced_to_full[kr])
        F[:, kr] += torch.tensordot(c, pair(k, k), dims=([0], [0]))
        for k2 in range(s.nk):
            v = pair(k, k2)
            for sp in range(s.ns):
                F[sp, kr] += pref * ((v @ D[k2, sp]) @ v.mH).sum(0)
    return F


def exact(case, seed):
    kind = case["kind"]
    if kind == "zgemm":
        A, B = _zgemm_inputs(case, seed)
        return A @ B
    if kind == "batch":
        return [_exact_gw(*_inputs(c, 100 * seed + i), False) for i, c in enumerate(_systems(case))]
    s, V = _inputs(case, seed)
    if kind == "hf":
        return _exact_fock(s, V)
    if kind == "scf":
        return _exact_fock(s, V), _exact_gw(s, V, False)
    return _exact_gw(s, V, bool(case.get("x2c")))
