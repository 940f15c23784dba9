"""Which products bem200_gemm accepts on which engine: complex64 from 128 rows, 64
columns, k = 64 and 2^26 multiply-adds needs a workspace on engine 1 and is
refused on engine 2; what is smaller, and complex128, runs without.  The
workspace may start at any address."""
import ctypes

import numpy as np
import pytest

from mnpbem_b200 import _native as nat

pytestmark = pytest.mark.gpu

ERR_ARG, ERR_UNSUPPORTED = 1, 4


def _call(dt, engine, m, n, k, wsb=0, offset=0):
    """(status, relative error against numpy in double)"""
    import torch
    rng = np.random.default_rng(m + n + k)
    A = (rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))).astype(dt)
    B = (rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))).astype(dt)
    At, Bt = torch.as_tensor(A, device="cuda"), torch.as_tensor(B, device="cuda")
    Ct = torch.zeros((m, n), dtype=At.dtype, device="cuda")
    ws = torch.empty(wsb + offset + 16, dtype=torch.uint8, device="cuda") if wsb else None
    wp = ctypes.c_void_p(ws.data_ptr() + offset) if wsb else None
    al, be = (ctypes.c_double * 2)(1.0, 0.0), (ctypes.c_double * 2)(0.0, 0.0)
    code = nat.C128 if dt == np.complex128 else nat.C64
    st = nat.lib().bem200_gemm(code, engine, m, n, k, al, nat.ptr(At), k, nat.ptr(Bt), n, be, nat.ptr(Ct), n, wp, wsb,
                               nat.stream_ptr())
    if st:
        return st, None
    ref = A.astype(np.complex128) @ B.astype(np.complex128)
    return 0, float(np.max(np.abs(Ct.cpu().numpy() - ref)) / np.max(np.abs(ref)))


# (64, 1100, 1000) and (100, 700, 1000) are below 128 rows; (1024, 1024, 63) below k = 64;
# (200, 200, 1000) below 2^26 multiply-adds
@pytest.mark.parametrize("engine", [1, 2])
@pytest.mark.parametrize("m,n,k", [(64, 1100, 1000), (100, 700, 1000), (1100, 1024, 63), (200, 200, 1000), (1100, 63, 1024)])
def test_small_complex64_products_need_no_workspace(cuda, engine, m, n, k):
    st, err = _call(np.complex64, engine, m, n, k)
    assert st == 0 and err < 1e-4, (st, err)


@pytest.mark.parametrize("m,n,k", [(128, 1024, 512), (1024, 1024, 64), (1500, 1500, 128)])
def test_large_complex64_products_are_refused_without(cuda, m, n, k):
    assert _call(np.complex64, 1, m, n, k)[0] == ERR_ARG
    assert _call(np.complex64, 2, m, n, k)[0] == ERR_UNSUPPORTED
    st, err = _call(np.complex64, 1, m, n, k, wsb=int(nat.lib().bem200_gemm_workspace_size(1, m, n, k)))
    assert st == 0 and err < 1e-5


@pytest.mark.parametrize("engine", [1, 2])
def test_complex128_products_need_no_workspace(cuda, engine):
    st, err = _call(np.complex128, engine, 512, 512, 512)
    assert st == 0 and err < 1e-13


@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
@pytest.mark.parametrize("offset", [0, 1, 4, 255])
def test_workspace_at_any_address(cuda, dt, offset):
    wsb = 3 * int(nat.lib().bem200_gemm_workspace_size(1, 500, 500, 500))
    st, err = _call(dt, 1, 500, 500, 500, wsb=wsb, offset=offset)
    assert st == 0 and err < (1e-6 if dt == np.complex64 else 1e-14), (st, err)
