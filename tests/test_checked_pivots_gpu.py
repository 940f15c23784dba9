"""The LU without row exchanges reports a needed exchange also when the pivot is
exactly zero: an identity with two rows exchanged, inside a 64-row block, across
its edge, and with the nonzero entry only below the block."""
import numpy as np
import pytest

from mnpbem_b200 import _native as nat

pytestmark = pytest.mark.gpu


def _factor(A, code):
    import torch
    n = A.shape[0]
    At = torch.as_tensor(A, device="cuda")
    rowmap, ipiv = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    wsb = int(nat.lib().bem200_getrf_workspace_size(code, 0, n))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    nat.call("bem200_getrf_ex", code, 0, n, nat.ptr(At), n, nat.ptr(rowmap), nat.ptr(ipiv), nat.ptr(info), nat.ptr(ws),
             wsb, 4, 0, nat.stream_ptr())
    return int(info.item())


@pytest.mark.parametrize("dt,code", [(np.complex64, nat.C64), (np.complex128, nat.C128)], ids=["c64", "c128"])
@pytest.mark.parametrize("n,i,j", [(64, 10, 40), (130, 10, 100), (130, 63, 64), (130, 0, 129), (700, 63, 699),
                                   (700, 200, 300), (1300, 640, 1299)])
def test_zero_pivot_that_needs_an_exchange(cuda, dt, code, n, i, j):
    A = np.eye(n, dtype=dt)
    assert _factor(A, code) == 0
    A[[i, j]] = A[[j, i]]
    assert _factor(A, code) == -nat.ERR_PIVOTING


@pytest.mark.parametrize("dt,code", [(np.complex64, nat.C64), (np.complex128, nat.C128)], ids=["c64", "c128"])
def test_zero_pivot_met_during_the_elimination(cuda, dt, code):
    """Column 63 of the first block cancels to an exact zero pivot; one entry
    below the block stays."""
    n = 200
    A = np.eye(n, dtype=dt)
    A[63, 0] = A[0, 63] = 1.0    # a_63,63 - a_63,0 a_0,63 = 0
    A[150, 63] = 0.25
    assert _factor(A, code) == -nat.ERR_PIVOTING
    A[150, 63] = 0.0             # nothing left to exchange with: a singular matrix, reported by its column
    assert _factor(A, code) == 64
