"""The panel kernels and the FP64 inverse levels at the sizes where they change: sub-panels
of 16 columns and 32 rows, one launch or two per diagonal block (the rows fill the GPU or
not), one or two streams, pairs of blocks of a level and a ragged last pair, k slabs; pivots
that are not normal positive numbers."""
from __future__ import annotations

import numpy as np
import pytest

import cucholesky as cc
from cucholesky import matgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [15, 16, 17, 31, 32, 33, 47, 48, 49, 111, 112, 113, 127, 128, 129, 144, 145, 159, 160,
                               161, 176, 192, 193, 240, 255, 256, 257, 288])
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("p", "sdcz")
def test_potrf_subpanel_edges(handle, p, uplo, n):
    A = matgen.spd(p, n, seed=n, lda=n + 1)
    D = cc.to_device_colmajor(A)
    assert cc.potrf(handle, D, n, uplo) == 0
    F = cc.to_host_colmajor(D)
    assert matgen.backward_error(A[:n], F[:n], uplo) <= 2.0
    keep = np.tril(np.ones((n, n), bool)) if uplo == "L" else np.triu(np.ones((n, n), bool))
    assert np.array_equal(F[:n][~keep], A[:n][~keep]) and np.array_equal(F[n:], A[n:])


@pytest.mark.parametrize("n", [1536, 1537, 4864, 4865, 5000])
@pytest.mark.parametrize("p,uplo", [("s", "L"), ("d", "U"), ("d", "L"), ("c", "U"), ("z", "L")])
def test_potrf_launch_limits(handle, p, uplo, n):
    # 1536: one stream; 4864 = 148 x 32 + 128: the rows below the first block fill the GPU
    import torch
    A = matgen.spd_device(p, n, seed=n)
    W = A.to(matgen.torch_dtype(p)).contiguous()
    H = matgen.hermitian_of(W, uplo)
    assert cc.potrf(handle, W, n, uplo) == 0
    assert matgen.probe_backward_error(H, matgen.factor_of(W, uplo), p) <= 1.0
    # a bad pivot in a block after the limit, and in the first one
    for k in (n - 40, 70):
        B = A.to(matgen.torch_dtype(p)).contiguous()
        B[k, k] = -1.0
        assert cc.potrf(handle, B, n, uplo) == k + 1
    torch.cuda.synchronize()


@pytest.mark.parametrize("p", "sdcz")
def test_info_at_every_column_of_a_subpanel(handle, p):
    n = 150
    A = matgen.spd(p, n, seed=3)
    F = A.copy(order="F")
    D = cc.to_device_colmajor(F)
    assert cc.potrf(handle, D, n) == 0
    good = cc.to_host_colmajor(D)
    eps = np.finfo(matgen.dtype_of(p)).eps
    for k in list(range(16, 33)) + [127, 128, 129, 149]:
        for bad in (-1.0, 0.0, np.nan):
            B = A.copy(order="F")
            B[k, k] = bad
            D = cc.to_device_colmajor(B)
            assert cc.potrf(handle, D, n) == k + 1
            # the columns before it within its 128-column block are factored
            c0 = k // 128 * 128 if p != "z" else k // 64 * 64
            got = cc.to_host_colmajor(D)[c0:k, c0:k]
            assert np.abs(np.tril(got - good[c0:k, c0:k])).max(initial=0) <= 200 * eps


@pytest.mark.parametrize("p", "dz")
def test_subnormal_and_large_pivots(handle, p):
    n = 40
    A = matgen.spd(p, n, seed=9)
    L = np.linalg.cholesky(A)
    for s in (2.0 ** -1030, 2.0 ** 1018):
        D = cc.to_device_colmajor(np.asfortranarray(A * s))
        assert cc.potrf(handle, D, n) == 0
        F = np.tril(cc.to_host_colmajor(D))
        # the scaled matrix itself holds 2^-44 of relative precision when it is subnormal
        assert np.abs(F / np.sqrt(s) - L).max() <= (2.0 ** -38 if s < 1 else 1e-13)


@pytest.mark.parametrize("n", [129, 192, 257, 383, 385, 513, 640, 769, 1025, 1100])
@pytest.mark.parametrize("p,uplo", [("d", "L"), ("d", "U"), ("z", "L"), ("z", "U")])
def test_fp64_inverse_levels_and_slabs(handle, p, uplo, n):
    A = matgen.spd(p, n, seed=n)
    L = np.linalg.cholesky(A)
    T0 = L if uplo == "L" else L.conj().T
    keep = np.tril(np.ones((n, n), bool)) if uplo == "L" else np.triu(np.ones((n, n), bool))
    bound = 2.0 ** -53 * (32 + np.sqrt(n))
    for pad in (0, 1, 2):
        T = np.full((n + pad, n), 7.0, dtype=T0.dtype, order="F")
        T[:n][keep] = T0[keep]
        W = np.where(keep, T[:n], 0)
        for call, ref in ((cc.trtri, np.linalg.inv(W)), (cc.lauum, W.conj().T @ W if uplo == "L" else W @ W.conj().T)):
            D = cc.to_device_colmajor(T)
            assert call(handle, D, n, uplo) == 0
            got = cc.to_host_colmajor(D)
            d = np.where(keep, got[:n] - ref, 0)
            assert np.linalg.norm(d) <= bound * np.linalg.norm(np.where(keep, ref, 0))
            assert np.array_equal(got[:n][~keep], T[:n][~keep]) and np.array_equal(got[n:], T[n:])


@pytest.mark.parametrize("uplo", "LU")
def test_batched_fp32_edges(handle, uplo):
    import torch
    sizes = [1, 2, 15, 16, 17, 31, 33, 63, 64, 65, 100, 127, 128, 129, 191, 192, 193, 256, 257, 300]
    mats = [matgen.spd("s", n, seed=n) for n in sizes]
    bad = 11
    mats[bad] = mats[bad].copy(order="F")
    mats[bad][70, 70] = -1.0
    flat, off, _ = cc.pack_colmajor(mats, np.float32)
    buf = torch.from_numpy(flat.copy()).cuda()
    plan = cc.BatchedPlan(handle, buf, sizes, off, uplo=uplo, flags=7)
    for _ in range(2):
        buf.copy_(torch.from_numpy(flat))
        plan.run()
        info, logdet = plan.results()
        out = buf.cpu().numpy()
        for b, (n, m, o) in enumerate(zip(sizes, mats, off)):
            if b == bad:
                assert info[b] == 71
                continue
            assert info[b] == 0
            A = m.astype(np.float64)
            assert abs(logdet[b] - np.linalg.slogdet(A)[1]) <= 100 * n * 2.0 ** -23
            inv = np.linalg.inv(A)
            got = out[o:o + n * n].reshape(n, n).T
            keep = np.tril(np.ones((n, n), bool)) if uplo == "L" else np.triu(np.ones((n, n), bool))
            assert np.linalg.norm(np.where(keep, got - inv, 0)) <= 2.0 ** -24 * (32 + np.sqrt(n)) * np.linalg.norm(inv)
            assert np.array_equal(got[~keep], m[~keep])
    plan.close()


@pytest.mark.parametrize("nrhs", [1, 3, 4, 5, 8, 9, 16, 17])
@pytest.mark.parametrize("uplo", "LU")
def test_potrs_right_hand_side_groups(handle, uplo, nrhs):
    import torch
    for n in (1, 63, 64, 65, 200, 449):
        A = matgen.spd("d", n, seed=n)
        D = cc.to_device_colmajor(A)
        assert cc.potrf(handle, D, n, uplo) == 0
        B = np.random.default_rng(n).standard_normal((n, nrhs))
        X = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
        rc, info = cc.call_potrs(handle, "D", uplo, n, nrhs, D.data_ptr(), n, X.data_ptr(), n)
        assert rc == 0 and info == 0
        ref = np.linalg.solve(A, B)
        assert np.linalg.norm(X.cpu().numpy().T - ref) <= 2.0 ** -53 * 8 * (32 + np.sqrt(n)) * np.linalg.norm(ref)


@pytest.mark.parametrize("prec", [cc.MIXED_BF16, cc.MIXED_TF32])
@pytest.mark.parametrize("n,nrhs,uplo", [(127, 1, "L"), (128, 1, "L"), (129, 2, "U"), (255, 3, "L"), (641, 16, "U"),
                                         (2047, 5, "L"), (2048, 1, "U"), (2049, 16, "L"), (2400, 17, "L"),
                                         (4864, 2, "U"), (4865, 2, "L"), (6200, 3, "L")])
def test_mixed_launch_limits(handle, prec, n, nrhs, uplo):
    """The mixed factor's panels (the block and its rows in one launch while they fit the
    GPU, 4864 = 148 x 32 + 128) and the preconditioner's products (2048-wide steps, their
    triangular blocks, split or not): W W^T against S A S + shift I to the rounding of the
    operands, and the refined solution to the criterion that ends the refinement."""
    import torch
    A = matgen.spd_device("d", n, seed=n).contiguous()
    H = matgen.hermitian_of(A, uplo)
    plan = cc.MixedPlan(handle, uplo, n, A.data_ptr(), n, prec)
    assert plan.info == 0
    w, ldw, s, anorm, shift = plan.factor()
    torch.cuda.synchronize()

    def view(ptr, count, typestr):
        raw = type("Raw", (), {"__cuda_array_interface__": {"shape": (count,), "typestr": typestr,
                                                            "data": (ptr, False), "version": 2}})
        return torch.as_tensor(raw(), device="cuda").clone()
    L = torch.tril(view(w, n * ldw, "<f4").reshape(n, ldw)[:, :n].T).double()
    S = view(s, n, "<f8")
    M = S[:, None] * H * S[None, :] + shift * torch.eye(n, dtype=torch.float64, device="cuda")
    # every product rounds two operands to u: |E| <= 2u |L| |L|^T, whose Frobenius norm is at
    # most |L|_F^2 = trace(M) <= sqrt(n) |M|_F; the roundings are independent, so sqrt(n) u falls
    # to a small multiple of u
    u = 2.0 ** -8 if prec == cc.MIXED_BF16 else 2.0 ** -11
    assert float(torch.linalg.norm(M - L @ L.T) / torch.linalg.norm(M)) <= 4 * u
    B = torch.as_tensor(np.random.default_rng(n).standard_normal((nrhs, n)), device="cuda")
    X = torch.zeros_like(B)
    it, berr = plan.solve(nrhs, B.data_ptr(), n, X.data_ptr(), n)
    tol = np.sqrt(n) * 2.0 ** -53
    assert it > 0 and berr <= tol
    R = torch.abs(B - X @ H).amax(1) / (torch.abs(H).sum(1).max() * torch.abs(X).amax(1) + torch.abs(B).amax(1))
    assert float(R.max()) <= 2 * tol
    plan.close()
