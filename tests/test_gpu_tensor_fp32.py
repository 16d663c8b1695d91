"""FP32 ?trtri, ?lauum, ?potri and ?potrf on the TF32 tensor cores (real and complex, any
alignment): the tile and level edges (orders around 256, 384, 512 and odd ones, one and
several pairs per level, a last pair of one row), both storages and diagonals, against
FP64 numpy; and the range rule: entries outside it give exactly what the SIMT engine
gives."""
from __future__ import annotations

import os

import numpy as np
import pytest

import cucholesky as cc
from cucholesky import matgen

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24
ORDERS = [256, 257, 300, 383, 385, 511, 513, 641, 897, 1025]


def _tri(p, n, uplo, seed, pad):
    """A well-conditioned triangular factor with the other triangle and padding set to a sentinel."""
    A = matgen.spd(p, n, seed=seed).astype(np.complex128 if p == "c" else np.float64)
    L = np.linalg.cholesky(A)
    T = L if uplo == "L" else L.conj().T
    out = np.full((n + pad, n), 7.0, dtype=matgen.dtype_of(p), order="F")
    keep = np.tril(np.ones((n, n), bool)) if uplo == "L" else np.triu(np.ones((n, n), bool))
    out[:n, :n] = np.where(keep, T, 7.0).astype(out.dtype)
    return out, keep


def _wide(a):
    return a.astype(np.complex128 if np.iscomplexobj(a) else np.float64)


def _check(got, ref, before, keep, bound):
    n = ref.shape[0]
    g = _wide(got[:n, :n])
    d = np.where(keep, g - ref, 0)
    assert np.linalg.norm(d) <= bound * np.linalg.norm(np.where(keep, ref, 0))
    assert np.array_equal(got[:n, :n][~keep], before[:n, :n][~keep]) and np.array_equal(got[n:], before[n:])


@pytest.mark.parametrize("n", ORDERS)
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("p", "sc")
def test_trtri_lauum_against_fp64(handle, p, uplo, n):
    # rounding errors of sums of up to n terms, twice, times the condition number (about 3)
    bound = EPS * (32 + np.sqrt(n))
    for pad, diag in ((0, "N"), (1, "U"), (3, "N")):
        T, keep = _tri(p, n, uplo, n, pad)
        W = _wide(np.where(keep, T[:n, :n], 0))
        if diag == "U":
            # a unit triangle whose inverse does not grow: off-diagonal entries scaled by 1 / n
            T[:n, :n] = np.where(keep, (T[:n, :n] / n).astype(T.dtype), 7.0)
            T[np.arange(n), np.arange(n)] = 5.0
            W = _wide(np.where(keep, T[:n, :n], 0))
            np.fill_diagonal(W, 1.0)
        D = cc.to_device_colmajor(T)
        assert cc.trtri(handle, D, n, uplo, diag) == 0
        ref = np.linalg.inv(W)
        offdiag = keep & ~np.eye(n, dtype=bool) if diag == "U" else keep
        _check(cc.to_host_colmajor(D), ref, T, offdiag, bound)
        if diag == "N":
            D = cc.to_device_colmajor(T)
            assert cc.lauum(handle, D, n, uplo) == 0
            ref = W.conj().T @ W if uplo == "L" else W @ W.conj().T
            _check(cc.to_host_colmajor(D), ref, T, keep, bound)
            if p == "c":
                assert not np.any(np.imag(cc.to_host_colmajor(D)[np.arange(n), np.arange(n)]))


@pytest.mark.parametrize("n", [129, 255, 385, 700, 1025])
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("p", "sc")
def test_potrf_any_alignment(handle, p, uplo, n):
    for pad in (0, 1, 2, 4):
        A = matgen.spd(p, n, seed=n, lda=n + pad)
        D = cc.to_device_colmajor(A)
        assert cc.potrf(handle, D, n, uplo) == 0
        F = cc.to_host_colmajor(D)
        assert matgen.backward_error(A[:n], F[:n], uplo) <= 1.0
        keep = np.tril(np.ones((n, n), bool)) if uplo == "L" else np.triu(np.ones((n, n), bool))
        assert np.array_equal(F[:n][~keep], A[:n][~keep]) and np.array_equal(F[n:], A[n:])
        B = A.copy(order="F")
        k = n - 3
        B[k, k] = -1.0
        D = cc.to_device_colmajor(B)
        assert cc.potrf(handle, D, n, uplo) == k + 1


@pytest.mark.parametrize("bad", [np.inf, np.nan, 2.0 ** 70, "tiny"])
@pytest.mark.parametrize("p", "sc")
def test_range_rule_matches_simt(handle, p, bad):
    os.environ["CUCHOLESKY_FORCE_SIMT"] = "1"
    try:
        simt = cc.Handle()
    finally:
        del os.environ["CUCHOLESKY_FORCE_SIMT"]
    n = 300
    T, _ = _tri(p, n, "L", 5, 0)
    if bad == "tiny":
        T = np.asfortranarray((T * np.float32(2.0 ** -70)).astype(T.dtype))
    else:
        T[200, 50] = bad
    for call in (cc.trtri, cc.lauum):
        out = []
        for h in (handle, simt):
            D = cc.to_device_colmajor(T)
            assert call(h, D, n, "L") == 0
            out.append(cc.to_host_colmajor(D))
        assert np.array_equal(out[0], out[1], equal_nan=True)
    simt.close()
