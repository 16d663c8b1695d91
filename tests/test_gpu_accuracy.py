"""Rounding errors of the panel kernels and of the split TF32 products, against wider
arithmetic: the diagonal and the column scaling of a pivot, the updates inside a diagonal
block, and the FP32 inverse against the plain FP32 engine's."""
from __future__ import annotations

import os

import numpy as np
import pytest

import cucholesky as cc
from cucholesky import matgen

pytestmark = pytest.mark.gpu

U = {"s": 2.0 ** -24, "d": 2.0 ** -53, "c": 2.0 ** -24, "z": 2.0 ** -53}


def _matrix(p, n, seed):
    """G G^H / n + I, rounded to the type; its diagonal and its pivots lie about 1 and 2."""
    rng = np.random.default_rng(seed)
    G = rng.uniform(-1, 1, (n, n)) if p in "sd" else (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(2)
    return np.asfortranarray((G @ G.conj().T / n + np.eye(n)).astype(matgen.dtype_of(p)))


def _wide_factor(A):
    """The lower factor in at least 11 more bits than A's type."""
    if A.dtype in (np.float32, np.complex64):
        return np.linalg.cholesky(A.astype(np.complex128 if np.iscomplexobj(A) else np.float64))
    L = A.astype(np.clongdouble if np.iscomplexobj(A) else np.longdouble)
    n = L.shape[0]
    for j in range(n):
        d = np.sqrt(L[j, j].real)
        L[j, j] = d
        L[j + 1:, j] /= d
        L[j + 1:, j + 1:] -= np.outer(L[j + 1:, j], L[j + 1:, j].conj())
    return np.tril(L)


@pytest.mark.parametrize("p,n", [("s", 100), ("s", 129), ("s", 300), ("d", 16), ("d", 100), ("c", 100), ("c", 129),
                                 ("c", 300), ("z", 16), ("z", 60)])
@pytest.mark.parametrize("uplo", "LU")
def test_factor_rounding(handle, p, n, uplo):
    # An element takes one subtraction per 16 columns and at most 16 more inside its own, so in
    # a 128-column block 12 roundings on average, each of rms u / sqrt(3) times a value below 2;
    # the diagonal elements, which are most of the norm, get half of that, at most
    # 0.5 sqrt(12) 2 u / sqrt(3) = 2 u and with pivots spread over 1 .. 2 about 1.4 u.  (64
    # roundings, one per column, give sqrt(64 / 12) times as much; measured 1.8 to 2.4 u, and
    # 0.9 to 1.1 u so.)
    err = []
    for seed in range(4):
        A = _matrix(p, n, seed)
        D = cc.to_device_colmajor(A)
        assert cc.potrf(handle, D, n, uplo) == 0
        F = cc.to_host_colmajor(D)
        F = np.tril(F) if uplo == "L" else np.triu(F).conj().T
        L = _wide_factor(A)
        err.append(np.linalg.norm((F - L).astype(np.complex128)) / np.linalg.norm(L.astype(np.complex128)))
    assert np.mean(err) <= 1.4 * U[p]


@pytest.mark.parametrize("n", [100, 256])
@pytest.mark.parametrize("p", "sd")
def test_pivot_roots(handle, p, n):
    """Blocks [[d, b], [b, c]]: L11 = sqrt(d) and L21 = b / sqrt(d) for random mantissas, even
    and odd exponents and both ends of the normal range."""
    real, wide, u = (np.float32, np.float64, U["s"]) if p == "s" else (np.float64, np.longdouble, U["d"])
    fi = np.finfo(real)
    # a rounded root's reciprocal scales the column: u from the reciprocal (FP32: the hardware's
    # estimate, documented to 2^-22.9) and u from the product; FP64's Taylor step drops 2^-58
    bound = (2.0 ** -22.9 + u) if p == "s" else 2.05 * u
    rng = np.random.default_rng(n)
    exps = np.concatenate([np.arange(fi.minexp, fi.minexp + 8), np.arange(fi.maxexp - 8, fi.maxexp),
                           rng.integers(fi.minexp, fi.maxexp, 12 * (n // 2))])
    for k in range(0, len(exps) - n // 2, n // 2):
        e = exps[k:k + n // 2]
        d = np.ldexp(rng.uniform(1, 2, n // 2).astype(wide), e).astype(real)
        b = (np.sqrt(d.astype(wide)) * rng.uniform(0.5, 1, n // 2)).astype(real)
        A = np.zeros((n, n), real, order="F")
        i = np.arange(0, n, 2)
        A[i, i], A[i + 1, i], A[i, i + 1], A[i + 1, i + 1] = d, b, b, 4
        D = cc.to_device_colmajor(A)
        assert cc.potrf(handle, D, n) == 0
        F = cc.to_host_colmajor(D)
        assert np.array_equal(F[i, i], np.sqrt(d))
        ref = b.astype(wide) / np.sqrt(d.astype(wide))
        assert np.max(np.abs(F[i + 1, i].astype(wide) / ref - 1)) <= bound
        assert np.count_nonzero(np.tril(F, -1)) == n // 2


@pytest.mark.parametrize("n", [257, 300, 384, 513, 1000])
@pytest.mark.parametrize("p", "sc")
def test_split_inverse_no_worse_than_simt(handle, p, n):
    """?potri of the same factor on the TF32 tensor cores and on the FP32 engine: the split
    products' sums, rounded to nearest every 32 k, err no more than one FMA chain per element."""
    os.environ["CUCHOLESKY_FORCE_SIMT"] = "1"
    try:
        simt = cc.Handle()
    finally:
        del os.environ["CUCHOLESKY_FORCE_SIMT"]
    err = {}
    for seed in range(3):
        L = np.linalg.cholesky(_matrix(p, n, seed).astype(np.complex128 if p == "c" else np.float64))
        T = np.asfortranarray(L.astype(matgen.dtype_of(p)))
        W = np.linalg.inv(T.astype(L.dtype))
        ref = np.tril(W.conj().T @ W)
        for name, h in (("split", handle), ("simt", simt)):
            D = cc.to_device_colmajor(T)
            assert cc.potri(h, D, n) == 0
            got = np.tril(cc.to_host_colmajor(D)).astype(L.dtype)
            err.setdefault(name, []).append(np.linalg.norm(got - ref) / np.linalg.norm(ref))
    simt.close()
    assert np.mean(err["split"]) <= 1.05 * np.mean(err["simt"]), err


@pytest.mark.parametrize("p,n,uplo", [("s", 4095, "L"), ("s", 4200, "U"), ("c", 2047, "U"), ("c", 2100, "L")])
def test_split_inverse_of_long_sums(handle, p, n, uplo):
    """On either side of the order from which an accumulator takes two k blocks (4096 real k):
    the inverse errs less than the FP32 engine's."""
    import torch
    os.environ["CUCHOLESKY_FORCE_SIMT"] = "1"
    try:
        simt = cc.Handle()
    finally:
        del os.environ["CUCHOLESKY_FORCE_SIMT"]
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    G = torch.randn((n, n), generator=g, device="cuda", dtype=torch.complex128 if p == "c" else torch.float64)
    A = G @ G.conj().T / n + torch.eye(n, device="cuda", dtype=G.dtype)
    T = torch.tril(torch.linalg.cholesky(A)).to(matgen.torch_dtype(p))     # the lower factor, [i, j]
    ref = torch.cholesky_inverse(T.to(G.dtype))
    # storage [j, i] = A(i, j): the lower factor for L, its conjugate transpose for U
    stored = (T.T if uplo == "L" else T.conj()).resolve_conj().contiguous()
    keep = torch.triu if uplo == "L" else torch.tril
    want = keep(ref.T)
    err = []
    for h in (handle, simt):
        D = stored.clone()
        assert cc.potri(h, D, n, uplo) == 0
        torch.cuda.synchronize()
        err.append(float(torch.linalg.norm(keep(D).to(G.dtype) - want) / torch.linalg.norm(want)))
    simt.close()
    assert err[0] <= err[1], err
