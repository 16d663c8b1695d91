"""Calls at the limits of the kernels they would take: ranges of FP32 entries, memory that is
refused or tight, failing pivots on either side of a launch rule."""
from __future__ import annotations

import os

import numpy as np
import pytest

import cucholesky as cc
from cucholesky import matgen

pytestmark = pytest.mark.gpu


U = {"s": 2.0 ** -24, "d": 2.0 ** -53}


@pytest.fixture(scope="module")
def simt():
    """A handle whose products all run on the plain FP32 engine."""
    os.environ["CUCHOLESKY_FORCE_SIMT"] = "1"
    try:
        h = cc.Handle()
    finally:
        del os.environ["CUCHOLESKY_FORCE_SIMT"]
    yield h
    h.close()


def _factor_error(A, F, uplo):
    """|F - L| / |L| against FP64 (A and F as numpy arrays of an FP32 type)."""
    w = np.complex128 if np.iscomplexobj(A) else np.float64
    L = np.linalg.cholesky(A.astype(w))
    F = np.tril(F) if uplo == "L" else np.triu(F).conj().T
    return np.linalg.norm(F.astype(w) - L) / np.linalg.norm(L)


# Split products lose what falls below 2^-126: entries about 2^-110 are where that shows
# first (3e-6), entries above 2^126 overflow.  Both take the FP32 engine, bit for bit.
@pytest.mark.parametrize("case", ["small", "one small row", "large", "infinite"])
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("p,uplo,n", [("s", "L", 300), ("s", "U", 700), ("c", "L", 300), ("c", "U", 700)])
def test_potrf_range_rule(handle, simt, p, uplo, n, pad, case):
    A = matgen.spd(p, n, seed=n)
    A = A / np.abs(np.diag(A)).max()
    if case == "one small row":
        A[n // 2] *= np.float32(2.0 ** -55)
        A[:, n // 2] *= np.float32(2.0 ** -55)
    elif case == "small":
        A = A * np.float32(2.0 ** -110)
    elif case == "large":
        A = A * np.float32(2.0 ** 127)
    else:
        A[n // 2, n // 2] = np.inf
    T = np.zeros((n + pad, n), A.dtype, order="F")
    T[:n] = A
    out = []
    for h in (handle, simt):
        D = cc.to_device_colmajor(T)
        info = cc.potrf(h, D, n, uplo)
        out.append((info, cc.to_host_colmajor(D)))
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1], equal_nan=True)
    if case in ("small", "large"):
        assert out[0][0] == 0 and _factor_error(A, out[0][1][:n], uplo) <= 4 * 2.0 ** -24
    # a failing pivot is found all the same
    k = n - 5
    B = T.copy(order="F")
    B[k, k] = -1.0
    if case != "infinite":
        assert cc.potrf(handle, cc.to_device_colmajor(B), n, uplo) == k + 1


@pytest.mark.parametrize("scale", [2.0 ** -79, 2.0 ** 125])
@pytest.mark.parametrize("p,n", [("s", 301), ("c", 300)])
def test_potrf_split_products_within_range(handle, p, n, scale):
    """Just inside the range the error is that of the unscaled matrix (powers of two are exact)."""
    A = matgen.spd(p, n, seed=n)
    A = (A / np.abs(np.diag(A)).max()).astype(A.dtype)   # the diagonal at most 1
    A[np.arange(n), np.arange(n)] = np.maximum(np.diag(A).real, 0.5)
    err = []
    for s in (1.0, scale):
        D = cc.to_device_colmajor(np.asfortranarray((A * s).astype(A.dtype)))
        assert cc.potrf(handle, D, n) == 0
        err.append(_factor_error(A * s if s == 1.0 else (A * s).astype(A.dtype), cc.to_host_colmajor(D), "L"))
    assert err[1] <= 1.1 * err[0] + 2.0 ** -26


@pytest.mark.parametrize("memory", ["pinned", "device"])
@pytest.mark.parametrize("p,uplo", [("s", "U"), ("c", "L")])
def test_host_potrf_range_rule(p, uplo, memory):
    """The streamed host-memory factor (n >= 2048: a panel, then the rest) of small entries."""
    import torch
    n = 2100
    A = matgen.spd(p, n, seed=4)
    A = (A * np.float32(2.0 ** -110)).astype(A.dtype)
    T = torch.from_numpy(np.ascontiguousarray(A.T))
    T = T.pin_memory() if memory == "pinned" else T.cuda()
    gpus = cc.MultiGPU([0])
    hh = cc.HostHandle(gpus)
    rc, info = cc.call_host(hh, p.upper(), "potrf", uplo, n, T.data_ptr(), n)
    torch.cuda.synchronize()
    assert rc == 0 and info == 0
    assert _factor_error(A, T.cpu().numpy().T, uplo) <= 4 * 2.0 ** -24


def _refuse_allocation(after):
    import ctypes as C
    f = cc.lib().cuLAPACKFailAllocation
    f.argtypes, f.restype = [C.c_int], C.c_int
    assert f(after) == 0


@pytest.mark.parametrize("p,pad", [("c", 0), ("s", 1)])
def test_potrf_without_memory_for_the_splits(simt, p, pad):
    """The operand splits take more memory than the panel: refused, the call still succeeds."""
    n = 300
    T = matgen.spd(p, n, seed=6, lda=n + pad)
    h = cc.Handle()
    D, S = cc.to_device_colmajor(T), cc.to_device_colmajor(T)
    _refuse_allocation(0)
    try:
        assert cc.potrf(h, D, n) == 0
    finally:
        _refuse_allocation(-1)
    assert cc.potrf(simt, S, n) == 0
    assert np.array_equal(cc.to_host_colmajor(D), cc.to_host_colmajor(S))
    h.close()


def _held_after(call):
    """Device memory that a fresh handle holds after call(handle)."""
    import torch
    h = cc.Handle()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    call(h)
    torch.cuda.synchronize()
    held = free0 - torch.cuda.mem_get_info()[0]
    h.close()
    return held


@pytest.mark.parametrize("p,n,limit", [("s", 8193, 0.75), ("d", 8193, 0.65), ("c", 16385, 6.5)])
def test_trtri_memory_with_a_last_pair_of_one_row(p, n, limit):
    """One row past a power of two: the buffers of the last level are as narrow as its last
    pair (GiB held by the handle; FP64 with 0.5 for an aligned copy), and the inverse is
    right, also where the level's columns come in pieces (complex, above 8 GiB)."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    t = matgen.torch_dtype(p)
    T = torch.randn((n, n), generator=g, device="cuda", dtype=t).div_(n)
    T.diagonal().copy_(torch.rand(n, generator=g, device="cuda").add_(1))
    X = T.clone()
    held = _held_after(lambda h: cc.trtri(h, X, n))
    assert held <= limit * 2 ** 30, held / 2 ** 30
    wide = torch.complex128 if p == "c" else torch.float64
    v = torch.randn((4, n), generator=g, device="cuda", dtype=wide)
    w = v
    for S in (X, T):                    # [j, i] = A(i, j): the lower triangle of A
        w = w @ S.triu_().T.to(wide)
    err = float(torch.linalg.norm(w - v) / torch.linalg.norm(v))
    assert err <= {"s": 2.0 ** -20, "c": 2.0 ** -20, "d": 2.0 ** -48}[p], err


def test_mixed_solve_when_its_workspace_is_refused():
    """The plan's block inverses are formed for fewer blocks at a time."""
    import torch
    n = 4300
    A = matgen.spd_device("d", n, seed=2).contiguous()
    B = torch.randn((3, n), device="cuda", dtype=torch.float64)
    X = torch.zeros_like(B)
    for after in (1, 2, 3):
        h = cc.Handle()
        _refuse_allocation(after)
        try:
            rc, it, berr, info = cc.call_posv_mixed(h, "L", n, 3, A.data_ptr(), n, B.data_ptr(), n, X.data_ptr(), n)
        finally:
            _refuse_allocation(-1)
        if rc == 0:
            break
        h.close()
    assert rc == 0 and info == 0
    R = B - X @ matgen.hermitian_of(A, "L")
    assert float(R.abs().max()) <= 1e-11
    h.close()


@pytest.mark.parametrize("p,n", [("z", 1100), ("c", 1000), ("d", 1100)])
def test_first_potri_grows_the_workspace_once(p, n):
    """A second growth would be refused here, and the product then take another route."""
    L = np.linalg.cholesky(matgen.spd(p, n, seed=8).astype(np.complex128 if p in "cz" else np.float64))
    T = np.asfortranarray(L.astype(matgen.dtype_of(p)))
    out = []
    for after in (1, -1):
        h = cc.Handle()
        D = cc.to_device_colmajor(T)
        _refuse_allocation(after)
        try:
            assert cc.potri(h, D, n) == 0
        finally:
            _refuse_allocation(-1)
        out.append(np.tril(cc.to_host_colmajor(D)))
        h.close()
    assert np.array_equal(out[0], out[1])


def _batch(p, n, batch):
    import torch
    mats = [matgen.spd(p, n, seed=b) for b in range(batch)]
    flat, off, sizes = cc.pack_colmajor(mats, matgen.dtype_of(p))
    return mats, torch.from_numpy(flat).cuda(), off, sizes


@pytest.mark.parametrize("p", "sd")
@pytest.mark.parametrize("flags,nb", [(7, 0), (7, 32), (3, 0), (7, -1)])
def test_batched_plan_memory(p, flags, nb):
    """Two matrices of order 3000: the plan holds the inverse's workspace and little more, not
    inverse blocks for CTAs that never run."""
    import torch
    n = 3000
    h = cc.Handle()
    buf = torch.zeros(2 * n * n, dtype=matgen.torch_dtype(p), device="cuda")
    for o in (0, n * n):
        buf[o:o + n * n].view(n, n).fill_diagonal_(1.0)
    plans = []

    def create(_):
        plans.append(cc.BatchedPlan(h, buf, [n, n], [0, n * n], flags=flags, nb=nb))
    held = _held_after(create)
    work = 2 * n * n * buf.element_size() if flags & 4 else 0
    assert held <= work + (48 << 20), held >> 20
    plans[0].run()
    info, _ = plans[0].results()
    assert info == [0, 0]
    plans[0].close()
    h.close()


@pytest.mark.parametrize("after", [4, 5])
@pytest.mark.parametrize("p", "sd")
def test_batched_plan_without_the_persistent_workspace(p, after):
    """Refused, the tuner chooses among the grouped forms."""
    mats, buf, off, sizes = _batch(p, 200, 5)
    h = cc.Handle()
    _refuse_allocation(after)
    try:
        plan = cc.BatchedPlan(h, buf, sizes, off, flags=7, nb=0)
    finally:
        _refuse_allocation(-1)
    assert plan.nb in (32, 64)
    plan.run()
    info, logdet = plan.results()
    for b, A in enumerate(mats):
        inv = np.linalg.inv(A.astype(np.float64))
        got = buf[off[b]:off[b] + 200 * 200].view(200, 200).T.cpu().numpy()
        assert info[b] == 0
        assert np.linalg.norm(np.tril(got - inv)) <= {"s": 2.0 ** -18, "d": 2.0 ** -47}[p] * np.linalg.norm(inv)
    plan.close()
    h.close()


def _check_inverse(A, got, uplo, u):
    n = A.shape[0]
    inv = np.linalg.inv(A.astype(np.float64))
    keep = np.tril(np.ones((n, n), bool)) if uplo == "L" else np.triu(np.ones((n, n), bool))
    # condition numbers of about 3: rounding errors of sums of up to n terms
    assert np.linalg.norm(np.where(keep, got - inv, 0)) <= u * (32 + np.sqrt(n)) * np.linalg.norm(inv), n
    assert np.array_equal(got[~keep], A[~keep])


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("flags", [7, 3])
@pytest.mark.parametrize("p", "sd")
def test_batched_persistent_form(handle, p, flags, uplo):
    """nb = -1 for both types: matrices at the edges of the 64 x 64 tiles, one that fails, and
    the factor alone."""
    import torch
    sizes = [1, 2, 16, 63, 64, 65, 127, 128, 129, 200, 256, 257, 500]
    mats = [matgen.spd(p, n, seed=n) for n in sizes]
    mats[9] = mats[9].copy(order="F")
    mats[9][150, 150] = -1.0
    flat, off, _ = cc.pack_colmajor(mats, matgen.dtype_of(p))
    buf = torch.from_numpy(flat.copy()).cuda()
    plan = cc.BatchedPlan(handle, buf, sizes, off, uplo=uplo, flags=flags, nb=-1)
    assert plan.nb == -1 and plan.form == -1
    for _ in range(2):
        buf.copy_(torch.from_numpy(flat))
        plan.run()
        info, logdet = plan.results()
        out = buf.cpu().numpy()
        for b, (n, A, o) in enumerate(zip(sizes, mats, off)):
            if b == 9:
                assert info[b] == 151
                continue
            got = out[o:o + n * n].reshape(n, n).T
            assert info[b] == 0
            assert abs(logdet[b] - np.linalg.slogdet(A.astype(np.float64))[1]) <= 200 * n * U[p]
            if flags & 4:
                _check_inverse(A, got, uplo, U[p])
            else:
                assert matgen.backward_error(A, np.asfortranarray(got), uplo) <= 2
    plan.close()


@pytest.mark.parametrize("p", "sd")
def test_batched_form_makes_the_plan_again(handle, p):
    mats, buf, off, sizes = _batch(p, 130, 40)
    plan = cc.BatchedPlan(handle, buf, sizes, off, flags=7, nb=0)
    again = cc.BatchedPlan(handle, buf, sizes, off, flags=7, nb=plan.form)
    assert again.form == plan.form and plan.form in (-1, 32, 64)
    assert plan.nb == plan.form or (p == "s" and plan.nb == 64)
    again.close()
    plan.close()


@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("p", "sdcz")
def test_contents_after_a_bad_pivot(handle, p, uplo):
    """The columns before the bad pivot hold the factor, the others of its block what they held:
    with rows below the block (one launch) and without (the block alone)."""
    nb = 64 if p == "z" else 128
    A = matgen.spd(p, 300, seed=12)
    A = A if uplo == "L" else np.asfortranarray(A.conj().T)
    for n in (nb, 300):
        for k in (0, 5, 20, 31, 47, nb - 1):
            G = A[:n, :n].copy(order="F")
            D = cc.to_device_colmajor(G)
            assert cc.potrf(handle, D, n, uplo) == 0
            good = cc.to_host_colmajor(D)
            B = G.copy(order="F")
            B[k, k] = -1.0
            D = cc.to_device_colmajor(B)
            assert cc.potrf(handle, D, n, uplo) == k + 1
            got = cc.to_host_colmajor(D)
            if uplo == "U":
                got, good, B = got.T, good.T, B.T
            low = np.tril(np.ones((n, nb), bool))
            done = low & (np.arange(nb) < k)
            # up to the pivot's own row the factor does not depend on it (but for rounding: a
            # sub-panel with a bad pivot goes through a plain loop)
            rest = np.arange(n) != k
            d = np.abs(np.where(done, got[:, :nb] - good[:, :nb], 0))[rest]
            assert d.max() <= 64 * np.finfo(got.real.dtype).eps
            assert np.array_equal(got[:, :nb][low & ~done], B[:, :nb][low & ~done])


@pytest.mark.parametrize("n", [40, 128])
@pytest.mark.parametrize("p", "sc")
def test_subnormal_and_large_fp32_pivots(handle, p, n):
    """Pivots below 2^-126 hold fewer bits (2^-149 apart), those near 2^127 all of them."""
    A = matgen.spd(p, n, seed=n)
    A = A / np.abs(np.diag(A)).max()
    for scale, bound in ((2.0 ** -130, 2.0 ** -19 * n), (2.0 ** 127, 4 * U["s"])):
        B = (A * np.float32(scale)).astype(A.dtype)
        D = cc.to_device_colmajor(B)
        assert cc.potrf(handle, D, n) == 0
        assert _factor_error(B, cc.to_host_colmajor(D), "L") <= bound


@pytest.mark.parametrize("bad", [np.inf, np.nan, 2.0 ** 70, "tiny"])
@pytest.mark.parametrize("p", "sc")
def test_inverse_range_rule(handle, simt, p, bad):
    """?trtri and ?lauum of entries that the splits cannot hold, at an order where either type
    would take them: the FP32 engine's results, bit for bit."""
    n = 400
    T = np.tril(np.linalg.cholesky(matgen.spd(p, n, seed=5))).astype(matgen.dtype_of(p), order="F")
    if bad == "tiny":
        T = np.asfortranarray(T * np.float32(2.0 ** -70))
    else:
        T[250, 50] = bad
    for call in (cc.trtri, cc.lauum):
        out = []
        for h in (handle, simt):
            D = cc.to_device_colmajor(T)
            assert call(h, D, n, "L") == 0
            out.append(cc.to_host_colmajor(D))
        assert np.array_equal(out[0], out[1], equal_nan=True)
