"""Tensor-core GEMM in residue arithmetic (engine 1) against long-double numpy,
within the bound of its operand rounding: with scaled norms of at least
2^25.5 (complex64) / 2^57 (complex128) and half a unit of rounding per real
component, |dC_ij| <= 2 (sqrt(2 k) / 2) |a_i| |b_j| / (that norm), besides a few
roundings of the result."""
import ctypes

import numpy as np
import pytest

from mnpbem_b200 import _native as nat

pytestmark = pytest.mark.gpu

NORM = {np.complex64: 2.0 ** 25.5, np.complex128: 2.0 ** 57}


def _rand(rng, n, m, dt):
    return (rng.standard_normal((n, m)) + 1j * rng.standard_normal((n, m))).astype(dt)


def _gemm(A, B, C, alpha, beta, ws_bytes=None):
    import torch
    m, k = A.shape
    n = B.shape[1]
    code = nat.C128 if A.dtype == np.complex128 else nat.C64
    At, Bt, Ct = (torch.as_tensor(x, device="cuda") for x in (A, B, C))
    if ws_bytes is None:
        ws_bytes = int(nat.lib().bem200_gemm_workspace_size(1, m, n, k)) * (1 if code == nat.C64 else 3)
    ws = torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")
    al, be = (ctypes.c_double * 2)(alpha.real, alpha.imag), (ctypes.c_double * 2)(beta.real, beta.imag)
    nat.call("bem200_gemm", code, 1, m, n, k, al, nat.ptr(At), k, nat.ptr(Bt), n, be, nat.ptr(Ct), n, nat.ptr(ws),
             ws_bytes, nat.stream_ptr())
    torch.cuda.synchronize()
    return Ct.cpu().numpy()


def _check(A, B, C, got, alpha, beta):
    dt = A.dtype.type
    k = A.shape[1]
    P = A.astype(np.clongdouble) @ B.astype(np.clongdouble)
    ref = alpha * P + beta * C.astype(np.clongdouble)
    na = np.sqrt(np.sum(np.abs(A.astype(np.clongdouble)) ** 2, axis=1))
    nb = np.sqrt(np.sum(np.abs(B.astype(np.clongdouble)) ** 2, axis=0))
    bound = np.sqrt(2 * k) * abs(alpha) * np.outer(na, nb) / NORM[dt]
    eps = np.finfo(A.real.dtype).eps
    bound = bound + 8 * eps * (abs(alpha) * np.abs(P) + abs(beta) * np.abs(C))
    assert np.all(np.abs(got - ref) <= bound), float(np.max(np.abs(got - ref) / bound))


# tile edges (128 rows, 256 columns, 128 k), remainders, one K pass and two
# (k > 3072), a product of few tiles and one of several tile rows
@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
@pytest.mark.parametrize("m,n,k", [(64, 1030, 1024), (128, 256, 2048), (129, 257, 2049), (700, 300, 333),
                                   (127, 255, 3201), (1290, 513, 129)])
def test_gemm_rns_edges(cuda, dt, m, n, k):
    rng = np.random.default_rng(m + n + k)
    A, B, C = _rand(rng, m, k, dt), _rand(rng, k, n, dt), _rand(rng, m, n, dt)
    A *= np.logspace(-6, 6, m)[:, None].astype(A.real.dtype)   # rows and columns of very different scales
    B *= np.logspace(4, -4, n)[None, :].astype(A.real.dtype)
    A[:, k // 2] *= 50
    al, be = -1.0 + 0.5j, 0.25 - 1.0j
    _check(A, B, C, _gemm(A, B, C, al, be), al, be)


@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
def test_gemm_rns_small_workspace_blocks(cuda, dt):
    """A workspace below the whole product's runs it in blocks of m and n (same
    bits: scales belong to rows and columns)."""
    rng = np.random.default_rng(5)
    m, n, k = 600, 700, 320
    A, B, C = _rand(rng, m, k, dt), _rand(rng, k, n, dt), _rand(rng, m, n, dt)
    full = _gemm(A, B, C, 1.0 + 0j, 1.0 + 0j)
    need = int(nat.lib().bem200_gemm_workspace_size(1, m, n, k)) * (1 if dt == np.complex64 else 3)
    small = _gemm(A, B, C, 1.0 + 0j, 1.0 + 0j, ws_bytes=need * 2 // 5)
    assert np.array_equal(full, small)


@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
def test_gemm_rns_special_values(cuda, dt):
    """Zero rows give exact zeros, rows and columns with an infinity or a NaN
    give NaN there and nowhere else, beta = 0 does not read C, and entries near
    the ends of the type's range keep their accuracy."""
    rng = np.random.default_rng(7)
    m, n, k = 260, 280, 1024
    A, B = _rand(rng, m, k, dt), _rand(rng, k, n, dt)
    big = 1e30 if dt == np.complex64 else 1e250
    A[3] = 0
    A[10] *= big
    A[11] /= big
    A[20, 5] = np.nan
    A[21, 6] = np.inf
    B[:, 9] = 0
    B[7, 30] = np.inf
    C = np.full((m, n), np.nan, dtype=dt)
    got = _gemm(A, B, C, 1.0 + 0j, 0j)
    assert np.all(got[3, :30] == 0) and np.all(np.delete(got[:, 9], [20, 21]) == 0)
    bad = np.zeros((m, n), bool)
    bad[[20, 21]] = True
    bad[:, 30] = True
    assert np.all(np.isnan(got[bad])) and np.all(np.isfinite(got[~bad]))
    rows, cols = np.delete(np.arange(m), [20, 21]), np.delete(np.arange(n), 30)
    A, B, got = A[rows], B[:, cols], got[np.ix_(rows, cols)]
    _check(A, B, np.zeros_like(got), got, 1.0, 0.0)
