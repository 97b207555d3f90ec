"""Timed cases of the framework's public entry points, and the same results in plain 64-bit torch or numpy.

A case is a dict of plain values; ``kind`` says which entry point it calls:

* ``matvec``  one H_eff theta.  ``path`` "operator" is what an eigensolver does (a ``MatVecMPOS`` kept, one ``MultAx`` per
  pass), "function" is the stateless ``matrix_vector_product``; ``engine`` picks FP64 (DMMA), the INT8-emulated FP64
  products or the split-BF16 mixed matvec of the operator.
* ``env``     one left or right environment update after a site was optimised (``env_update``).
* ``split``   the two-site Schmidt split (``schmidt_multisite``) and the truncated state U S V that the sweep goes on with.
* ``eigs``    one local ground-state solve (``MatVecMPOS.eigs``) from a start vector.
* ``fdmrg``   a whole two-site ground-state run (``fdmrg``) of a disordered Ising chain.

Tensors are column-major as in the library, so a torch tensor with the dims reversed holds the same bytes.
"""
import math

import numpy as np
import torch

import dmrg_b200 as hb

# Dense-count FLOPs of the largest listed matvec (complex, chi = 1024, D = 3, two sites); drawn matvecs stay below it.
_MATVEC_MOST = 4 * (16 * 3 * 1024**3 + 32 * 9 * 1024**2)


def listed():
    return [
        # the smallest solves of a sweep (chain ends, warm-up sweeps at bond 16): launches and latency
        dict(name="matvec op f64 16", kind="matvec", path="operator", engine="fp64", cplx=False, S=4, chiL=16, chiR=16, D=3),
        # the headline product: complex two-site H_eff at chi = 1024
        dict(name="matvec op c128 1024", kind="matvec", path="operator", engine="fp64", cplx=True, S=4, chiL=1024, chiR=1024, D=3),
        # a folded-spectrum product (H squared, D = 9) on the odd bonds that a truncation leaves
        dict(name="matvec op f64 D9 367x251", kind="matvec", path="operator", engine="fp64", cplx=False, S=4, chiL=367, chiR=251, D=9),
        # the contraction function on a one-site tensor of ordinary size
        dict(name="matvec fn c128 site 96x128", kind="matvec", path="function", engine="fp64", cplx=True, S=2, chiL=96, chiR=128, D=3),
        # the Krylov phase's product of a mixed-precision solve
        dict(name="matvec mixed c128 512", kind="matvec", path="operator", engine="mixed", cplx=True, S=4, chiL=512, chiR=512, D=3),
        # the opt-in FP64-accurate engine on a large bond that is no multiple of a tile
        dict(name="matvec int8 f64 1000", kind="matvec", path="operator", engine="int8", cplx=False, S=4, chiL=1000, chiR=1000, D=3),
        # environments of a right-moving (complex, H) and a left-moving (real, H squared, odd bonds) sweep
        dict(name="env L c128 256", kind="env", side="L", cplx=True, chiL=256, chiR=256, D=3),
        dict(name="env R f64 D9 640x517", kind="env", side="R", cplx=False, chiL=640, chiR=517, D=9),
        # a wide two-site split of moderate size, and the split of a chi = 256 sweep
        dict(name="split c128 35x86", kind="split", cplx=True, chiL=35, chiR=86),
        dict(name="split f64 256", kind="split", cplx=False, chiL=256, chiR=256),
        # one local solve of a sweep at a moderate bond
        dict(name="eigs f64 48", kind="eigs", cplx=False, chiL=48, chiR=48),
        # a whole ground-state calculation
        dict(name="fdmrg L16 chi32", kind="fdmrg", L=16, chi=32, sweeps=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bonds(rng, lo, hi):
    """Two neighbouring bonds: spread over their logarithm, equal one time in three, else up to a factor of two apart."""
    a = _log(rng, lo, hi)
    b = a if rng.random() < 1 / 3 else min(hi, max(lo, int(a * rng.uniform(0.5, 2.0))))
    return a, b


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "matvec", "env", "env", "split", "split", "eigs", "fdmrg"])
    cplx = rng.random() < 0.5
    if kind == "matvec":
        engine = rng.choice(["fp64", "fp64", "fp64", "int8", "mixed"])
        while True:
            a, b = _bonds(rng, 16 if engine == "fp64" else 128, 1024)
            S, D = rng.choice([2, 4]), rng.choice([3, 3, 9])
            c = dict(kind=kind, path=rng.choice(["operator", "function"]) if engine == "fp64" else "operator", engine=engine, cplx=cplx, S=S,
                     chiL=a, chiR=b, D=D)
            if work(c)["flops"] <= _MATVEC_MOST:
                return c
    if kind == "env":
        a, b = _bonds(rng, 16, 1024)
        return dict(kind=kind, side=rng.choice(["L", "R"]), cplx=cplx, chiL=a, chiR=b, D=rng.choice([3, 9]))
    if kind == "split":
        a, b = _bonds(rng, 12, 128 if cplx else 256)
        return dict(kind=kind, cplx=cplx, chiL=a, chiR=b)
    if kind == "eigs":
        a, b = _bonds(rng, 16, 64)
        return dict(kind=kind, cplx=cplx, chiL=a, chiR=b)
    return dict(kind=kind, L=rng.randrange(12, 17), chi=_log(rng, 16, 32), sweeps=2)


# ------------------------------------------------------------------------------------------------------------ inputs
def _randn(g, *shape, cplx):
    return torch.randn(*shape, dtype=torch.complex128 if cplx else torch.float64, device="cuda", generator=g)


def _env(g, chi, D, cplx):
    """An environment block, entries of order 1/sqrt(chi), as [m, a', a]: every slice Hermitian, for D = 9 (H squared,
    m = i + 3 j) with the (i, j) <-> (j, i) pairing that the squared operator has."""
    E = _randn(g, D, chi, chi, cplx=cplx) / math.sqrt(chi)
    pair = torch.arange(D, device="cuda") if D != 9 else torch.arange(9, device="cuda").reshape(3, 3).T.reshape(-1)
    return ((E + E[pair].transpose(1, 2).conj()) / 2).contiguous()


def _fields(g, n):
    return (0.5 + torch.rand(n, dtype=torch.float64, device="cuda", generator=g)).cpu().numpy()


def _site_mpo(h, D, cplx):
    """Random-field Ising site MPO [D, D, 2, 2], or the uncompressed square of it (D = 9)."""
    W = np.zeros((3, 3, 2, 2))
    W[0, 0] = W[2, 2] = np.eye(2)
    W[1, 0] = np.diag([1.0, -1.0])
    W[2, 0] = [[0.0, -h], [-h, 0.0]]
    W[2, 1] = np.diag([-1.0, 1.0])
    if D == 9:
        W = np.einsum("mnsp,MNpt->mMnNst", W, W).reshape(9, 9, 2, 2, order="F")
    return np.asfortranarray(W.astype(np.complex128 if cplx else np.float64))


def _merged(sites):
    if len(sites) == 1:
        return sites[0]
    A, B = sites
    X = np.einsum("mcst,cnuv->mnsutv", A, B)
    return np.asfortranarray(X.reshape(A.shape[0], B.shape[1], 4, 4, order="F"))


def _device(W):
    return torch.from_numpy(np.ascontiguousarray(W.ravel(order="F"))).cuda()


def _host(E):
    return E.cpu().numpy().transpose(2, 1, 0)


def _inputs(case, seed):
    """The tensors of a case on the GPU (dims reversed) and host MPOs, from the seed alone."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    k, cplx = case["kind"], case.get("cplx", False)
    if k in ("matvec", "eigs"):
        cL, cR, D, S = case["chiL"], case["chiR"], case.get("D", 3), case.get("S", 4)
        sites = [_site_mpo(h, D, cplx) for h in _fields(g, 1 if S == 2 else 2)]
        x = _randn(g, cR, cL, S, cplx=cplx)
        return dict(sites=sites, L=_env(g, cL, D, cplx), R=_env(g, cR, D, cplx), x=x / torch.linalg.vector_norm(x))
    if k == "env":
        cL, cR, D = case["chiL"], case["chiR"], case["D"]
        M = _randn(g, cR, cL, 2, cplx=cplx) / math.sqrt(2 * (cL if case["side"] == "L" else cR))
        return dict(sites=[_site_mpo(_fields(g, 1)[0], D, cplx)], M=M, E=_env(g, cL if case["side"] == "L" else cR, D, cplx))
    if k == "split":
        # a two-site state whose Schmidt values fall from 1 to 1e-13, as those of a sweep do
        m, n = 2 * case["chiL"], 2 * case["chiR"]
        r = min(m, n)
        Q1, _ = torch.linalg.qr(_randn(g, m, r, cplx=cplx))
        Q2, _ = torch.linalg.qr(_randn(g, n, r, cplx=cplx))
        s = torch.exp(-torch.arange(r, device="cuda", dtype=torch.float64) * (30.0 / r))
        s = s / torch.linalg.vector_norm(s)
        A = (Q1 * s) @ Q2.mH  # rows s1 + 2 a, columns s2 + 2 b
        return dict(A=A, theta=A.reshape(case["chiL"], 2, case["chiR"], 2).permute(2, 0, 3, 1).contiguous())  # [b, a, s2, s1]
    return dict(h=_fields(g, case["L"]), seed=seed % 1000)


def _half(case):
    return min(case["chiL"], case["chiR"])  # a sweep keeps its bond: half of the split's singular values


def prepare(case, seed):
    d, k = _inputs(case, seed), case["kind"]
    s = dict(case=case)
    if k == "matvec" and case["path"] == "function":
        W = _merged(d["sites"])
        s |= dict(x=d["x"], y=torch.empty_like(d["x"]), W=_device(W), wd=W.shape, L=d["L"], R=d["R"])
    elif k in ("matvec", "eigs"):
        mixed = case.get("engine") == "mixed"
        op = hb.MatVecMPOS(d["sites"], _host(d["L"]), _host(d["R"]), cplx=case["cplx"], precision=hb.PREC_MIXED if mixed else hb.PREC_FP64)
        if case.get("engine") == "int8":
            op.set_fp64_engine(hb.FP64_INT8)
        s |= dict(op=op, x=d["x"], y=torch.empty_like(d["x"]))
    elif k == "env":
        W = d["sites"][0]
        chi = case["chiR"] if case["side"] == "L" else case["chiL"]
        s |= dict(M=d["M"], E=d["E"], W=_device(W), wd=W.shape, out=torch.empty(case["D"], chi, chi, dtype=d["E"].dtype, device="cuda"))
    elif k == "split":
        s |= dict(theta=d["theta"])
    else:
        s |= d
    return s


def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "matvec":
        if c["path"] == "operator":
            return s["op"].MultAx(s["x"], s["y"])
        cL, cR, D = c["chiL"], c["chiR"], c["D"]
        return hb.matrix_vector_product(s["y"], s["x"], (c["S"], cL, cR), s["W"], s["wd"], s["L"], (cL, cL, D), s["R"], (cR, cR, D))
    if k == "env":
        chi = c["chiL"] if c["side"] == "L" else c["chiR"]
        return hb.env_update(c["side"], s["out"], s["E"], (chi, chi, c["D"]), s["M"], (2, c["chiL"], c["chiR"]), s["W"], s["wd"])
    if k == "split":
        # the factors are unique up to a phase per singular value only: the state that they make is the output
        m, n = 2 * c["chiL"], 2 * c["chiR"]
        U, S, V, r, err = hb.schmidt_multisite(s["theta"], 2, 2, c["chiL"], c["chiR"], rank_max=_half(c), trunc_lim=1e-12)
        V = V.view(c["chiR"], r, 2).transpose(0, 1).reshape(r, n)
        return dict(S=S, theta=(U.view(r, m).T * S) @ V, rank=r, err=err)
    if k == "eigs":
        e, _ = s["op"].eigs(x0=s["x"].view(-1), x_out=s["y"].view(-1), tol=1e-12)
        # the solver's vector with the phase of the start vector, as a sweep that follows its state takes it
        o = torch.vdot(s["y"].view(-1), s["x"].view(-1))
        return dict(e=np.array(e), x=s["y"] * (o / o.abs()))
    r = hb.fdmrg(s["h"], chi_max=c["chi"], sweeps=c["sweeps"], seed=s["seed"])
    return dict(energy=np.array(r["energy"]), energies=np.array(r["energy_per_sweep"]), entropy=r["entropy_mid"])


# ------------------------------------------------------------------------------------------------- 64-bit references
def _matvec(d, x):
    W = torch.from_numpy(np.ascontiguousarray(_merged(d["sites"]))).cuda()
    t1 = torch.einsum("mpa,bas->mpbs", d["L"], x)
    t2 = torch.einsum("mnst,mpbs->npbt", W, t1)
    return torch.einsum("nqb,npbt->qpt", d["R"], t2).contiguous()


def _lowest(d, x, steps=700):
    """Lowest eigenpair by Lanczos with full re-orthogonalisation."""
    shape, q = x.shape, x.reshape(-1)
    Q, al, be = [], [], []
    for i in range(min(steps, q.numel())):
        Q.append(q)
        w = _matvec(d, q.reshape(shape)).reshape(-1)
        al.append(float(torch.vdot(q, w).real))
        B = torch.stack(Q, 1) if i % 25 == 0 else torch.cat([B, q[:, None]], 1)
        for _ in range(2):
            w = w - B @ (B.mH @ w)
        be.append(float(torch.linalg.vector_norm(w)))
        if i % 25 == 24 or be[-1] < 1e-12:
            e, v = np.linalg.eigh(np.diag(al) + np.diag(be[:-1], 1) + np.diag(be[:-1], -1))
            if abs(be[-1] * v[-1, 0]) < 1e-13 * abs(e).max():
                break
        q = w / be[-1]
    e, v = np.linalg.eigh(np.diag(al) + np.diag(be[:-1], 1) + np.diag(be[:-1], -1))
    u = B @ torch.from_numpy(np.ascontiguousarray(v[:, 0])).cuda().to(B.dtype)
    return e[0], u.reshape(shape) / torch.linalg.vector_norm(u)


def exact(case, seed):
    d, k = _inputs(case, seed), case["kind"]
    if k == "matvec":
        return _matvec(d, d["x"])
    if k == "env":
        W, M, E = torch.from_numpy(np.ascontiguousarray(d["sites"][0])).cuda(), d["M"], d["E"]
        if case["side"] == "L":  # [n, b', b] = sum E[m, a', a] M[b, a, s] conj(M)[b', a', s'] W[m, n, s, s']
            t = torch.einsum("mpa,bas->mpbs", E, M)
            t = torch.einsum("mnst,mpbs->npbt", W, t)
            return torch.einsum("npbt,qpt->nqb", t, M.conj())
        t = torch.einsum("nqb,bas->nqas", E, M)
        t = torch.einsum("mnst,nqas->mqat", W, t)
        return torch.einsum("mqat,qpt->mpa", t, M.conj())
    if k == "split":
        U, S, V = np.linalg.svd(d["A"].cpu().numpy(), full_matrices=False)
        r = _half(case)
        err, S = float(np.linalg.norm(S[r:])), S[:r] / np.linalg.norm(S[:r])
        return dict(S=torch.from_numpy(S), theta=torch.from_numpy((U[:, :r] * S) @ V[:r]), rank=None, err=err)
    if k == "eigs":
        e, u = _lowest(d, d["x"])
        o = torch.vdot(u.reshape(-1), d["x"].reshape(-1))
        return dict(e=np.array(e), x=u * (o / o.abs()))
    # free fermions: E0 = -(sum of the singular values of the bidiagonal matrix of fields and couplings)
    B = np.diag(d["h"]) + np.diag(np.ones(case["L"] - 1), 1)
    return dict(energy=np.array(-np.linalg.svd(B, compute_uv=False).sum()), energies=None, entropy=None)


# ------------------------------------------------------------------------------------------------------ what it takes
def work(case):
    k = case["kind"]
    f, e = (4, 16) if case.get("cplx") else (1, 8)  # real FLOPs per real multiply-add pair, bytes per element
    if k == "fdmrg":  # per bond update ten products, one split and one environment at the bonds that the chain allows
        L, n = case["L"], 0
        for i in range(L - 1):
            a, b = (min(case["chi"], 2 ** min(j, L - j)) for j in (i, i + 2))
            n += 10 * 24 * a * b * (a + b) + 22 * (2 * min(a, b)) ** 3 + 12 * a * b * (a + b)
        return dict(bytes=2.0 * case["sweeps"] * 8 * 16 * L * case["chi"] ** 2, flops=2.0 * case["sweeps"] * n)
    a, b = case["chiL"], case["chiR"]
    if k in ("matvec", "eigs"):
        S, D = case.get("S", 4), case.get("D", 3)
        n = 30 if k == "eigs" else 1  # a local solve takes some tens of products
        return dict(bytes=e * (2.0 * S * a * b + D * (a * a + b * b)), flops=n * f * (2.0 * S * D * a * b * (a + b) + 2.0 * S * S * D * D * a * b))
    if k == "env":
        D, chi, out = case["D"], (a if case["side"] == "L" else b), (b if case["side"] == "L" else a)
        return dict(bytes=e * (2.0 * a * b + D * (chi * chi + out * out)), flops=f * (4.0 * D * a * b * (a + b) + 8.0 * D * D * a * b))
    m, n = 2 * max(a, b), 2 * min(a, b)
    return dict(bytes=e * 4.0 * a * b * 2, flops=f * (4.0 * m * n * n + 8.0 * n**3))
