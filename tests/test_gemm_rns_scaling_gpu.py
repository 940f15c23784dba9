"""Residue GEMM on operands graded along the summation index, (A D)(D^-1 B): its
error against long double, relative to sum_k |a_ik| |b_kj|, beside that of the
CUDA-core product (engine 0) on the same operands.  complex128: no larger than
FP64 accumulation.  complex64: random operands have about half the error of FP32
accumulation; powers of two balance a column of A against a row of B to within
a factor of two each, so at most four times the FP32 error is allowed (the
bf16x3 products that engine 1 once ran had more than sixty times)."""
import ctypes

import numpy as np
import pytest

from mnpbem_b200 import _native as nat

pytestmark = pytest.mark.gpu

FACTOR = {np.complex64: 4.0, np.complex128: 1.0}


def _rand(rng, n, m, dt):
    return (rng.standard_normal((n, m)) + 1j * rng.standard_normal((n, m))).astype(dt)


def _gemm(A, B, engine, part=1.0):
    import torch
    m, k = A.shape
    n = B.shape[1]
    code = nat.C128 if A.dtype == np.complex128 else nat.C64
    At, Bt = (torch.as_tensor(x, device="cuda") for x in (A, B))
    Ct = torch.full((m, n), float("nan"), dtype=At.dtype, device="cuda")
    wsb = int(part * nat.lib().bem200_gemm_workspace_size(1, m, n, k) * (1 if code == nat.C64 else 3))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    al, be = (ctypes.c_double * 2)(1.0, 0.0), (ctypes.c_double * 2)(0.0, 0.0)
    nat.call("bem200_gemm", code, engine, m, n, k, al, nat.ptr(At), k, nat.ptr(Bt), n, be, nat.ptr(Ct), n, nat.ptr(ws),
             wsb, nat.stream_ptr())
    return Ct.cpu().numpy()


def _error(A, B, got, rows):
    W = np.clongdouble
    ref = A[rows].astype(W) @ B.astype(W)
    scale = np.abs(A[rows]).astype(np.longdouble) @ np.abs(B).astype(np.longdouble)
    return float(np.max(np.abs(got[rows] - ref) / scale))


def _grading(kind, k, rng, dt):
    wide = 2.0 ** 60 if dt == np.complex64 else 2.0 ** 500
    return {"none": np.ones(k), "1e4": np.logspace(-2, 2, k), "1e8": np.logspace(-4, 4, k),
            "random": 10.0 ** rng.uniform(-4, 4, k), "range": np.geomspace(1 / wide, wide, k),
            "spike": np.where(np.arange(k) == k // 3, 1e8, 1.0)}[kind]


def _operands(kind, m, n, k, dt):
    rng = np.random.default_rng(m + n + k)
    A, B = _rand(rng, m, k, np.complex128), _rand(rng, k, n, np.complex128)
    d = _grading(kind, k, rng, dt)
    A, B = A * d, B / d[:, None]
    if kind in ("1e8", "random"):  # rows and columns of different scales besides
        A *= 10.0 ** rng.uniform(-3, 3, (m, 1))
        B *= 10.0 ** rng.uniform(-3, 3, (1, n))
    return A.astype(dt), B.astype(dt)


# one block, k in two passes, a ragged product, many tile rows
@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
@pytest.mark.parametrize("kind", ["none", "1e4", "1e8", "random", "range", "spike"])
@pytest.mark.parametrize("m,n,k", [(300, 290, 1030), (130, 260, 3201), (1029, 259, 257)])
def test_grading_along_the_sum(cuda, dt, kind, m, n, k):
    A, B = _operands(kind, m, n, k, dt)
    rows = np.random.default_rng(1).choice(m, 12, replace=False)
    e_rns, e_fma = (_error(A, B, _gemm(A, B, e), rows) for e in (1, 0))
    assert e_rns <= FACTOR[dt] * e_fma, (e_rns, e_fma)


@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
def test_blocks_of_columns_with_their_own_grading(cuda, dt):
    """A small workspace runs n in blocks; only the middle columns of B are graded, and
    A is not: no scaling suits all columns.  Columns and rows that are zero take
    part."""
    m, n, k = 384, 1400, 512
    rng = np.random.default_rng(8)
    A, B = _rand(rng, m, k, dt), _rand(rng, k, n, dt)
    d = np.logspace(-3, 3, k)
    B[:, 512:900] *= d[:, None].astype(B.real.dtype)
    A[:, 7] = 0
    B[9] = 0
    rows = np.arange(0, m, 37)
    full, small = _gemm(A, B, 1), _gemm(A, B, 1, part=0.4)
    e_fma = _error(A, B, _gemm(A, B, 0), rows)
    for got in (full, small):
        assert np.all(np.isfinite(got))
        # the bound in norms, which a compromise between the columns may exceed by a few bits
        na = np.linalg.norm(A.astype(np.complex128), axis=1)
        nb = np.linalg.norm(B.astype(np.complex128), axis=0)
        ref = A.astype(np.clongdouble) @ B.astype(np.clongdouble)
        bound = np.sqrt(2 * k) * np.outer(na, nb) / {np.complex64: 2.0 ** 25.5, np.complex128: 2.0 ** 57}[dt]
        bound = bound * 2.0 ** 5 + 8 * np.finfo(A.real.dtype).eps * np.abs(ref)
        assert np.all(np.abs(got - ref) <= bound)
    plain = np.r_[0:512, 900:n]
    assert _error(A, B[:, plain], small[:, plain], rows) <= FACTOR[dt] * 8 * e_fma


@pytest.mark.parametrize("n", [830, 1500])
def test_inverse_of_a_graded_matrix(cuda, n):
    """complex64 inverse with in-place tensor-core products of D M D^-1, D powers
    of two from 1 to 2^-26: the inverse is D M^-1 D^-1, with the residual bound of
    the ungraded matrix in the balanced scale."""
    import torch
    rng = np.random.default_rng(n)
    M = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n) + 4 * np.eye(n)
    M = M.astype(np.complex64)
    d = 2.0 ** -np.round(np.linspace(0, 26, n))
    At = torch.as_tensor((d[:, None] * M / d).astype(np.complex64), device="cuda")
    L = nat.lib()
    scr = torch.empty(int(L.bem200_inverse_nopiv_workspace_size(nat.C64, n)), dtype=torch.uint8, device="cuda")
    wsb = int(L.bem200_gemm_workspace_size(1, n, n, n // 2 + 64))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.call("bem200_inverse_nopiv", nat.C64, 1, n, nat.ptr(At), n, nat.ptr(ws), wsb, nat.ptr(scr), 1e300,
             nat.ptr(info), nat.stream_ptr())
    assert int(info.item()) == 0
    X = At.cpu().numpy().astype(np.complex128) / d[:, None] * d
    r = np.abs(X @ M.astype(np.complex128) - np.eye(n)).max()
    assert r < 16 * n * 2.0 ** -24, r
