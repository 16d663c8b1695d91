"""The work that users of this library have it do, as measurable cases.

Every case goes through the package's public calls on matrices of the shapes and
distributions the library documents (A = G G^H / n + I for single matrices, the
squared-exponential kernel for batches, D (G G^T / n + 1e-3 I) D for the mixed
solve).  The kinds:

  factor   ?potrf, then ?logdet of the factor: a Gaussian log density, small to large
  solve    ?potrf and ?potrs with a few right-hand sides
  inverse  ?potrf, ?logdet and ?potri: a precision matrix with its determinant
  batched  one plan over many small matrices of uneven sizes: factor, log det, inverse
  mixed    cuDposvMixed: an FP64 solve on a TF32 factor with FP64 refinement
  host     cuMultiGPU?potrf on a matrix in page-locked host memory

A matrix is overwritten by its factor or inverse, so a pass starts by copying the
caller's matrix into the working buffer, as a program that keeps A would.
"""
from __future__ import annotations

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cuda-cholesky_b200"))
import cucholesky as cc  # noqa: E402

TYPES = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}
EPS = {"s": 2.0 ** -24, "d": 2.0 ** -53, "c": 2.0 ** -24, "z": 2.0 ** -53}


def listed():
    return [
        # one covariance block inside a sampler's loop: launches and latency
        dict(name="factor_d_100", kind="factor", type="d", uplo="L", n=100, pad=0),
        # a regression's normal equations: odd order, upper storage, a few right-hand sides
        dict(name="solve_d_1001", kind="solve", type="d", uplo="U", n=1001, pad=2, nrhs=5),
        # the library's plain FP64 configuration: factor, log det and inverse at n = 2048
        dict(name="inverse_d_2048", kind="inverse", type="d", uplo="L", n=2048, pad=0),
        # the headline: one large FP64 factorization
        dict(name="factor_d_16384", kind="factor", type="d", uplo="L", n=16384, pad=0),
        # the same order in single precision, upper storage
        dict(name="factor_s_16384", kind="factor", type="s", uplo="U", n=16384, pad=0),
        # a single-precision precision matrix of an order that fills no tile
        dict(name="inverse_s_6001", kind="inverse", type="s", uplo="L", n=6001, pad=0),
        # complex types: signal-processing covariances, factor and inverse
        dict(name="inverse_c_4096", kind="inverse", type="c", uplo="L", n=4096, pad=0),
        dict(name="inverse_z_3000", kind="inverse", type="z", uplo="U", n=3000, pad=0),
        # many small kernel matrices of uneven sizes 8..512, both precisions
        dict(name="batched_d_2000", kind="batched", type="d", uplo="L", batch=2000, hi=512),
        dict(name="batched_s_2000", kind="batched", type="s", uplo="L", batch=2000, hi=512),
        # an FP64 solve with 16 right-hand sides on the low-precision tensor cores
        dict(name="mixed_d_8192", kind="mixed", type="d", uplo="L", n=8192, nrhs=16, k=0.0),
        # the matrix lives in host memory, as it does for a caller of the host-memory routines
        dict(name="host_d_4096", kind="host", type="d", uplo="L", n=4096),
    ]


#: (kind, type) -> smallest and largest order that is drawn.
RANGES = {
    ("factor", "d"): (16, 14000), ("factor", "s"): (16, 12000), ("factor", "c"): (16, 7000), ("factor", "z"): (16, 7000),
    ("solve", "d"): (16, 6000), ("solve", "s"): (16, 6000),
    ("inverse", "d"): (16, 6000), ("inverse", "s"): (16, 8192), ("inverse", "c"): (16, 6000), ("inverse", "z"): (16, 4500),
    ("mixed", "d"): (1500, 10000), ("host", "d"): (500, 6000),
}


def draw(rng):
    kind = rng.choice(["factor", "factor", "factor", "solve", "inverse", "inverse", "inverse", "inverse", "batched", "mixed", "host"])
    uplo = rng.choice("LU")
    if kind == "batched":
        return dict(kind=kind, type=rng.choice("ds"), uplo=uplo, batch=int(round(math.exp(rng.uniform(math.log(50), math.log(2000))))),
                    hi=rng.randint(64, 512))
    p = rng.choice([t for (k, t) in RANGES if k == kind])
    lo, hi = RANGES[(kind, p)]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.3:                      # orders that fill their tiles are common too
        n = max(lo, n // 64 * 64)
    case = dict(kind=kind, type=p, uplo=uplo, n=n)
    if kind in ("factor", "solve", "inverse"):
        case["pad"] = rng.choice([0, 0, 0, 1, 4, 32])
    if kind in ("solve", "mixed"):
        case["nrhs"] = rng.randint(1, 16)
    if kind == "mixed":
        case["k"] = round(rng.uniform(0.0, 1.0), 2)
    return case


# ---- inputs --------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _hpd(p, n, pad, seed):
    """A = G G^H / n + I, rounded to the routine's type, as the tensor T with T[j, i] = A(i, j)
    and `pad` unused rows below each column."""
    g = _gen(seed)
    if p in "sd":
        G = torch.rand((n, n), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    else:
        G = torch.randn((n, n), generator=g, device="cuda", dtype=torch.complex128)
    A = G @ G.conj().T / n
    A.diagonal().add_(1.0)
    if p in "cz":
        A.diagonal().imag.zero_()
    T = torch.full((n, n + pad), 7.0, device="cuda", dtype=TYPES[p])
    T[:, :n] = A.T
    return T


def _scaled(n, k, seed):
    G = torch.randn((n, n), generator=_gen(seed), device="cuda", dtype=torch.float64)
    A = G @ G.T / n
    A.diagonal().add_(1e-3)
    d = 10.0 ** (k * torch.arange(n, device="cuda", dtype=torch.float64) / max(n - 1, 1))
    return (A * d[:, None] * d[None, :]).contiguous()


def _rhs(p, n, nrhs, seed):
    return torch.randn((nrhs, n), generator=_gen(seed + 7919), device="cuda", dtype=TYPES[p])


def _sizes(case):
    """The batch's orders, uniform in 8..hi: a plan is made for one list of them."""
    g = torch.Generator()
    g.manual_seed(1000 * case["batch"] + case["hi"])
    return torch.randint(8, case["hi"] + 1, (case["batch"],), generator=g).tolist()


def _kernels(case, seed):
    """Squared-exponential kernel matrices on uniform points of the unit cube, packed; the
    nugget is what each precision can factor (1e-4 in FP64, 1e-2 in FP32)."""
    p, sizes = case["type"], _sizes(case)
    x = torch.rand((sum(sizes), 3), generator=_gen(seed), device="cuda", dtype=torch.float64)
    buf = torch.empty(sum(n * n for n in sizes), device="cuda", dtype=TYPES[p])
    nugget = 1e-4 if p == "d" else 1e-2
    at, off, offs = 0, 0, []
    for n in sizes:
        y = x[at:at + n]
        K = torch.exp((y[:, None, :] - y[None, :, :]).square().sum(-1) * (-1.0 / (2 * 0.3 ** 2)))
        K.diagonal().add_(nugget)
        buf[off:off + n * n] = K.reshape(-1)
        offs.append(off)
        at, off = at + n, off + n * n
    return sizes, offs, buf


def prepare(case, seed):
    kind, p = case["kind"], case["type"]
    s = dict(case=case, h=cc.Handle())
    if kind == "batched":
        sizes, offs, A = _kernels(case, seed)
        W = A.clone()
        s.update(A=A, W=W, plan=cc.BatchedPlan(s["h"], W, sizes, offs, uplo=case["uplo"], flags=7))
    elif kind == "mixed":
        n, nrhs = case["n"], case["nrhs"]
        s.update(A=_scaled(n, case["k"], seed), B=_rhs(p, n, nrhs, seed))
        s["X"] = torch.zeros_like(s["B"])
    elif kind == "host":
        A = _hpd(p, case["n"], 0, seed).cpu().pin_memory()
        gpus = cc.MultiGPU([0])
        s.update(A=A, W=A.clone().pin_memory(), gpus=gpus, hh=cc.HostHandle(gpus))
    else:
        s["A"] = _hpd(p, case["n"], case["pad"], seed)
        s["W"] = s["A"].clone()
        if kind == "solve":
            s["B"] = _rhs(p, case["n"], case["nrhs"], seed)
            s["X"] = s["B"].clone()
    return s


# ---- one pass ------------------------------------------------------------------------

def run(s):
    case, h = s["case"], s["h"]
    kind, uplo = case["kind"], case["uplo"]
    if kind == "batched":
        s["W"].copy_(s["A"])
        s["plan"].run()
        info, logdet = s["plan"].results()
        return {"inverse": s["W"], "logdet": torch.tensor(logdet, dtype=torch.float64), "info": torch.tensor(info)}
    if kind == "mixed":
        n, B, X = case["n"], s["B"], s["X"]
        rc, _, _, info = cc.call_posv_mixed(h, uplo, n, case["nrhs"], s["A"].data_ptr(), n, B.data_ptr(), n, X.data_ptr(), n)
        if rc != 0:
            raise cc.CuCholeskyError("cuDposvMixed", rc)
        return {"x": X, "info": info}
    if kind == "host":
        s["W"].copy_(s["A"])
        rc, info = cc.call_host(s["hh"], case["type"].upper(), "potrf", uplo, case["n"], s["W"].data_ptr(), case["n"])
        if rc != 0:
            raise cc.CuCholeskyError("cuMultiGPUDpotrf", rc)
        return {"factor": s["W"], "info": info}
    n, W = case["n"], s["W"]
    W.copy_(s["A"])
    info = cc.potrf(h, W, n, uplo)
    if kind == "factor":
        return {"factor": W, "info": info, "logdet": cc.logdet_of_factor(h, W, n)}
    if kind == "solve":
        X = s["X"]
        X.copy_(s["B"])
        rc, _ = cc.call_potrs(h, case["type"].upper(), uplo, n, case["nrhs"], W.data_ptr(), W.shape[1], X.data_ptr(), n)
        if rc != 0:
            raise cc.CuCholeskyError("cu?potrs", rc)
        return {"factor": W, "info": info, "x": X}
    logdet = cc.logdet_of_factor(h, W, n)
    info += cc.potri(h, W, n, uplo)
    return {"inverse": W, "info": info, "logdet": logdet}


# ---- what a pass cannot do without ---------------------------------------------------

def work(case):
    kind, p = case["kind"], case["type"]
    size = {"s": 4, "d": 8, "c": 8, "z": 16}[p]
    per = 4 if p in "cz" else 1                 # real operations of a complex one
    if kind == "batched":
        # orders uniform in 8..hi: their mean square and cube
        hi, m = case["hi"], case["batch"]
        sq = sum(n * n for n in range(8, hi + 1)) / (hi - 7)
        cu = sum(n ** 3 for n in range(8, hi + 1)) / (hi - 7)
        return {"bytes": int(m * sq * size * 2), "flops": int(m * cu)}
    n = case["n"]
    tri = n * (n + 1) // 2 * size
    if kind == "mixed":
        return {"bytes": tri + 2 * n * case["nrhs"] * size, "flops": n ** 3 // 3 + 2 * n * n * case["nrhs"]}
    if kind == "host":
        return {"bytes": 2 * tri, "flops": n ** 3 // 3}
    # the working copy of the whole matrix, then the triangle in and out
    nbytes = 2 * n * (n + case["pad"]) * size + 2 * tri
    flops = per * n ** 3 // 3
    if kind == "solve":
        nbytes += 4 * n * case["nrhs"] * size
        flops += 2 * n * n * case["nrhs"]
    if kind == "inverse":
        nbytes += 2 * tri
        flops += per * 2 * n ** 3 // 3
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    kind, p = case["kind"], case["type"]
    eps = EPS[p]
    if kind == "batched":
        # squared-exponential kernels: condition numbers of about 1e6 (nugget 1e-4) and 1e4 (1e-2);
        # measured 2e-11 (largest 1.2e-9) and 6.4e-5 (1.8e-3)
        return {"rel": 1e-10, "max": 5e-9} if p == "d" else {"rel": 2.5e-4, "max": 8e-3}
    if kind == "mixed":
        # a normwise backward error of sqrt(n) eps times the condition number 10^(3.6 + 2k) of this
        # family, which the stopping rule allows; measured a tenth of it
        return {"rel": min(1e-4, 10 ** (3.6 + 2 * case["k"]) * math.sqrt(case["n"]) * eps)}
    # condition numbers of about 5: rounding errors of sums of up to n terms.  Measured against
    # 64 bits (in 64-bit types against another library's 64 bits): 2 to 27 eps over the ranges.
    return {"rel": eps * (32 + math.sqrt(case["n"]))}


# ---- the same in 64 bits -------------------------------------------------------------

def _keep(T, n, R, uplo):
    """The FP64 copy of T whose `uplo` triangle holds R(i, j) at T[j, i]."""
    out = T.to(torch.complex128 if T.is_complex() else torch.float64)
    R = R.transpose(0, 1)
    out[:, :n] = (torch.triu(R) + torch.tril(out[:, :n], -1)) if uplo == "L" else (torch.tril(R) + torch.triu(out[:, :n], 1))
    return out


def exact(case, seed):
    kind, p, uplo = case["kind"], case["type"], case["uplo"]
    if kind == "batched":
        sizes, offs, A = _kernels(case, seed)
        out, logdet = A.to(torch.float64), []
        for n, o in zip(sizes, offs):
            K = out[o:o + n * n].view(n, n)
            L = torch.linalg.cholesky(K)
            logdet.append(2 * L.diagonal().log().sum())
            out[o:o + n * n] = _keep(K, n, torch.cholesky_inverse(L), uplo).reshape(-1)
        return {"inverse": out, "logdet": torch.stack(logdet).cpu(), "info": torch.zeros(len(sizes), dtype=torch.int64)}
    n = case["n"]
    if kind == "mixed":
        A, B = _scaled(n, case["k"], seed), _rhs(p, n, case["nrhs"], seed)
        return {"x": torch.cholesky_solve(B.T, torch.linalg.cholesky(A)).T.contiguous(), "info": 0}
    T = _hpd(p, n, case.get("pad", 0), seed)
    wide = torch.complex128 if T.is_complex() else torch.float64
    A = T[:, :n].to(wide).transpose(0, 1)
    L = torch.linalg.cholesky(A)
    R = L if uplo == "L" else L.conj().transpose(0, 1).resolve_conj()
    if kind == "host":
        return {"factor": _keep(T, n, R, uplo).cpu(), "info": 0}
    logdet = float(2 * L.diagonal().real.log().sum())
    if kind == "factor":
        return {"factor": _keep(T, n, R, uplo), "info": 0, "logdet": logdet}
    if kind == "solve":
        B = _rhs(p, n, case["nrhs"], seed).to(wide)
        return {"factor": _keep(T, n, R, uplo), "info": 0, "x": torch.cholesky_solve(B.T, L).T.contiguous()}
    inv = torch.cholesky_inverse(L)
    return {"inverse": _keep(T, n, inv, uplo), "info": 0, "logdet": logdet}
