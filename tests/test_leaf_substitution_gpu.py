"""complex128 triangular leaves on ill-conditioned triangles: the residual is that
of substitution, |b - T x| <= 4 n u |T| |x| elementwise (n complex multiply-adds
per element, each of at most 2 sqrt(2) u), whatever the condition of T.  The
right-hand side is T x0 with x0 of order one, so x is small beside |T^-1| |b|."""
import numpy as np
import pytest

from mnpbem_b200 import _native as nat

pytestmark = pytest.mark.gpu


def _triangle(n, seed, unit):
    """Upper triangular, condition above 1e7 within 64 rows: the off-diagonal
    entries of a row add up to more than twice its diagonal."""
    rng = np.random.default_rng(seed)
    U = -0.4 * np.ones((n, n)) * np.exp(0.2j * rng.standard_normal((n, n)))
    U = np.triu(U, 1)
    U[np.abs(np.subtract.outer(np.arange(n), np.arange(n))) >= 64] *= 1e-3
    d = np.ones(n) if unit else np.exp(0.3 * rng.standard_normal(n) + 1j * rng.standard_normal(n))
    return U + np.diag(d)


def _getrs(LU, B):
    import torch
    n, nrhs = B.shape
    L = nat.lib()
    LUt, Bt = torch.as_tensor(LU, device="cuda"), torch.as_tensor(B, device="cuda")
    rowmap = torch.arange(n, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    scr = torch.empty(int(L.bem200_getrs_workspace_size(nat.C128, n, nrhs)), dtype=torch.uint8, device="cuda")
    nat.call("bem200_getrs", nat.C128, 0, n, nrhs, nat.ptr(LUt), n, nat.ptr(rowmap), nat.ptr(Bt), nrhs, None, 0,
             nat.ptr(scr), nat.ptr(status), nat.stream_ptr())
    return Bt.cpu().numpy()


def _check(T, X, B):
    W = np.clongdouble
    r = np.abs(B.astype(W) - T.astype(W) @ X.astype(W))
    bound = 4 * T.shape[0] * 2.0 ** -53 * (np.abs(T) @ np.abs(X))
    assert np.all(r <= bound), float(np.max(r / bound))


# one leaf (ragged and full), several; 16 and 32 vectors per CTA
@pytest.mark.parametrize("n,nrhs", [(33, 20), (64, 17), (64, 2500), (130, 40)])
@pytest.mark.parametrize("lower", [False, True], ids=["upper", "unit_lower"])
def test_left_leaves(cuda, n, nrhs, lower):
    rng = np.random.default_rng(n + nrhs)
    U = _triangle(n, n, lower)
    T = U[::-1, ::-1].copy() if lower else U
    assert n < 64 or np.linalg.cond(U[:64, :64]) > 1e7
    B = T @ (rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs)))
    _check(T, _getrs(T, B), B)


@pytest.mark.parametrize("rows", [40, 3000])
def test_rows_below_an_ill_conditioned_block(cuda, rows):
    """The rows of a checked LU below its first 64 columns: L21 U11 = A21."""
    import torch
    rng = np.random.default_rng(rows)
    U, n = _triangle(64, 5, False), 64 + rows
    U *= 1.0 / np.abs(np.diag(U))[:, None]
    A = np.eye(n, dtype=complex) * 4
    A[:64, :64] = U
    A[64:, :64] = 0.3 * (rng.standard_normal((rows, 64)) + 1j * rng.standard_normal((rows, 64))) / 4 @ U
    At = torch.as_tensor(A, device="cuda")
    rowmap, ipiv = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    wsb = int(nat.lib().bem200_getrf_workspace_size(nat.C128, 0, n))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    nat.call("bem200_getrf_ex", nat.C128, 0, n, nat.ptr(At), n, nat.ptr(rowmap), nat.ptr(ipiv), nat.ptr(info),
             nat.ptr(ws), wsb, 4, 0, nat.stream_ptr())
    X = At.cpu().numpy()[64:, :64]
    _check(U.T, X.T, A[64:, :64].T)
