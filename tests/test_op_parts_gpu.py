"""The parts of the BEM operator as separate calls (bem200_op_prep, the products in
any row order, bem200_hmat_gather_rows, bem200_op_combine) against
bem200_bem_apply."""
import ctypes

import numpy as np
import pytest

from mnpbem_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npol", [1, 3])
def test_operator_from_its_parts(cuda, npol):
    import torch
    n, w = 93, 8 * npol
    g = torch.Generator(device="cuda").manual_seed(npol)
    rnd = lambda *s: torch.randn(s, dtype=torch.complex128, device="cuda", generator=g)
    G1, G2, H1, H2 = (rnd(n, n) for _ in range(4))
    x, b = rnd(8 * n * npol), rnd(8 * n * npol)
    nvec = torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=g)
    e1, e2 = (ctypes.c_double * 2)(-11.0, 1.2), (ctypes.c_double * 2)(1.77, 0.0)
    p1, p2 = ctypes.cast(e1, ctypes.c_void_p), ctypes.cast(e2, ctypes.c_void_p)
    k0, s = 0.011, nat.stream_ptr()
    perm = torch.randperm(n, generator=g, device="cuda").to(torch.int32)
    inv = torch.argsort(perm.long()).to(torch.int32)
    U = []
    for side in range(2):
        u, c = torch.empty((n, w), dtype=torch.complex128, device="cuda"), torch.empty((n, w), dtype=torch.complex128, device="cuda")
        nat.call("bem200_op_prep", n, npol, ctypes.c_void_p(x.data_ptr() + 16 * 4 * n * npol * side), 0, p1, p2, side,
                 nat.ptr(u), s)
        nat.call("bem200_hmat_gather_rows", n, w, nat.ptr(u), nat.ptr(perm), nat.ptr(c), s)
        assert torch.equal(c, u[perm.long()])
        U.append(c)
    Y = []
    for M, side in ((G1, 0), (G2, 1), (H1, 0), (H2, 1)):
        y = torch.empty((n, w), dtype=torch.complex128, device="cuda")
        c = (M[perm.long()][:, perm.long()] @ U[side]).contiguous()
        nat.call("bem200_hmat_gather_rows", n, w, nat.ptr(c), nat.ptr(inv), nat.ptr(y), s)
        Y.append(y)
    scr = torch.empty(int(nat.lib().bem200_bem_apply_workspace_size(n, npol)), dtype=torch.uint8, device="cuda")
    for rhs in (None, b):
        got, ref = torch.empty_like(x), torch.empty_like(x)
        nat.call("bem200_op_combine", n, npol, *[nat.ptr(y) for y in Y], nat.ptr(nvec), k0, nat.ptr(rhs), nat.ptr(got), s)
        nat.call("bem200_bem_apply", n, npol, nat.ptr(G1), nat.ptr(G2), nat.ptr(H1), nat.ptr(H2), 0, p1, p2, nat.ptr(nvec),
                 k0, nat.ptr(x), ctypes.c_void_p(x.data_ptr() + 16 * 4 * n * npol), nat.ptr(rhs), nat.ptr(ref),
                 nat.ptr(scr), s)
        # n products per element on either side, condition of the sums about sqrt(n)
        assert float((got - ref).abs().max()) <= 64 * n * 2.0 ** -53 * float(ref.abs().max())
