"""Pivots at the ends of the exponent range: the leaves of the inverse, the
checked LU and the pivoted panels use reciprocals that stay finite and accurate
up to the largest numbers.  (The reciprocal of 1.5 x 2^1023 is subnormal with 50
bits, of 1.5 x 2^127 with 21: a few units of those are allowed.)"""
import numpy as np
import pytest

from mnpbem_b200 import _native as nat

pytestmark = pytest.mark.gpu

CASES = [(np.complex64, 127, 2.0 ** -18), (np.complex64, -126, 2.0 ** -20), (np.complex128, 1023, 2.0 ** -47),
         (np.complex128, 1020, 2.0 ** -49), (np.complex128, -1022, 2.0 ** -49)]
IDS = ["c64_high", "c64_low", "c128_high", "c128_1020", "c128_low"]


def _matrix(n, dt, expo):
    """Dominant diagonal near 2^expo, entries 1/16 of it on every second superdiagonal place."""
    rng = np.random.default_rng(n)
    D = np.diag(np.exp(2j * np.pi * rng.random(n)) * rng.uniform(1.0, 1.4, n))
    A = D + np.tril(rng.standard_normal((n, n)), -1) / 64 + np.triu(rng.standard_normal((n, n)), 1) / 64
    return A, (np.ldexp(A.real, expo) + 1j * np.ldexp(A.imag, expo)).astype(dt)


@pytest.mark.parametrize("dt,expo,tol", CASES, ids=IDS)
def test_inverse_leaf(cuda, dt, expo, tol):
    import torch
    n = 9
    A, As = _matrix(n, dt, expo)
    code = nat.C64 if dt == np.complex64 else nat.C128
    At = torch.as_tensor(As, device="cuda")
    scr = torch.empty(int(nat.lib().bem200_inverse_nopiv_workspace_size(code, n)), dtype=torch.uint8, device="cuda")
    ws, info = torch.empty(1, dtype=torch.uint8, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.call("bem200_inverse_nopiv", code, 0, n, nat.ptr(At), n, nat.ptr(ws), 0, nat.ptr(scr), 1e300, nat.ptr(info),
             nat.stream_ptr())
    X = At.cpu().numpy().astype(np.complex128)
    X = np.ldexp(X.real, expo) + 1j * np.ldexp(X.imag, expo)
    assert np.max(np.abs(X - np.linalg.inv(A))) < 64 * tol


# (the pivoted complex64 panels square the pivot's magnitude: not for these ranges)
@pytest.mark.parametrize("dt,expo,tol,flags", [(*c, 4) for c in CASES] + [(*c, 0) for c in CASES[2:]],
                         ids=[i + "-checked" for i in IDS] + [i + "-pivoted" for i in IDS[2:]])
def test_lu_multipliers(cuda, dt, expo, tol, flags):
    import torch
    n = 70
    A, As = _matrix(n, dt, expo)
    code = nat.C64 if dt == np.complex64 else nat.C128
    At = torch.as_tensor(As, device="cuda")
    rowmap, ipiv = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    wsb = int(nat.lib().bem200_getrf_workspace_size(code, 0, n))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    nat.call("bem200_getrf_ex", code, 0, n, nat.ptr(At), n, nat.ptr(rowmap), nat.ptr(ipiv), nat.ptr(info), nat.ptr(ws),
             wsb, flags, 0, nat.stream_ptr())
    assert int(info.item()) == 0 and np.array_equal(rowmap.cpu().numpy(), np.arange(n))
    F = At.cpu().numpy().astype(np.complex128)
    U = np.triu(np.ldexp(F.real, -expo) + 1j * np.ldexp(F.imag, -expo))
    L = np.tril(F, -1) + np.eye(n)
    assert np.max(np.abs(L @ U - A)) < 64 * tol
