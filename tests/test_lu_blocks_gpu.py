"""Block edges of the complex128 LU without row exchanges (64-column diagonal
blocks, rows below multiplied by U11^-1) and of the 64-row triangular leaves
(32 x 32 inverses, 16 or 32 vectors per CTA), against numpy.  Tolerances: a
well-conditioned matrix (cond ~ 3), n eps growth: 1e-13 relative."""
import numpy as np
import pytest

from mnpbem_b200 import _native as nat

pytestmark = pytest.mark.gpu


def _dominant(n, seed):
    rng = np.random.default_rng(seed)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
    return A + 4 * np.eye(n)


# one ragged block, exact blocks, one column over, several blocks; few
# vectors, a ragged CTA of vectors, more than 148 x 16 (32 per CTA)
@pytest.mark.parametrize("n,nrhs", [(17, 33), (64, 17), (65, 40), (96, 2400), (129, 31), (200, 18), (321, 64)])
def test_checked_lu_and_triangular_leaves_c128(cuda, n, nrhs):
    import torch
    A = _dominant(n, n)
    B = np.random.default_rng(n + 1).standard_normal((n, nrhs)) + 1j
    L = nat.lib()
    At, Bt = torch.as_tensor(A, device="cuda"), torch.as_tensor(B, device="cuda")
    rowmap, ipiv = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    info, status = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
    wsb = int(L.bem200_getrf_workspace_size(nat.C128, 0, n))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    nat.call("bem200_getrf_ex", nat.C128, 0, n, nat.ptr(At), n, nat.ptr(rowmap), nat.ptr(ipiv), nat.ptr(info),
             nat.ptr(ws), wsb, 4, 0, nat.stream_ptr())
    assert int(info.item()) == 0
    F = At.cpu().numpy()
    P = (np.tril(F, -1) + np.eye(n)) @ np.triu(F)
    assert np.max(np.abs(P - A)) <= 1e-13 * np.max(np.abs(A)) * np.sqrt(n)
    scr = torch.empty(int(L.bem200_getrs_workspace_size(nat.C128, n, nrhs)), dtype=torch.uint8, device="cuda")
    nat.call("bem200_getrs", nat.C128, 0, n, nrhs, nat.ptr(At), n, nat.ptr(rowmap), nat.ptr(Bt), nrhs, nat.ptr(ws), wsb,
             nat.ptr(scr), nat.ptr(status), nat.stream_ptr())
    X = np.linalg.solve(A, B)
    assert np.max(np.abs(Bt.cpu().numpy() - X)) <= 1e-13 * np.max(np.abs(X)) * np.sqrt(n)


@pytest.mark.parametrize("dt,code,eps", [(np.complex64, nat.C64, 2.0 ** -24), (np.complex128, nat.C128, 2.0 ** -53)],
                         ids=["c64", "c128"])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 63, 64, 65, 67])
def test_inverse_leaf_edges(cuda, n, dt, code, eps):
    """The register Gauss-Jordan leaf at the edges of its 4 x 4 thread tiles
    and of the 64 x 64 block.  The matrix is diagonally dominant with condition
    number below 3, so the residual of the computed inverse stays below
    16 n eps (a few roundings per step, n steps)."""
    import torch
    A = _dominant(n, 40 + n).astype(dt)
    At = torch.as_tensor(A, device="cuda")
    scr = torch.empty(int(nat.lib().bem200_inverse_nopiv_workspace_size(code, n)), dtype=torch.uint8, device="cuda")
    ws = torch.empty(1, dtype=torch.uint8, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.call("bem200_inverse_nopiv", code, 0, n, nat.ptr(At), n, nat.ptr(ws), 0, nat.ptr(scr), 1e-2,
             nat.ptr(info), nat.stream_ptr())
    assert int(info.item()) == 0
    X = At.cpu().numpy().astype(np.complex128)
    r = np.abs(X @ A.astype(np.complex128) - np.eye(n)).max()
    assert r < 16 * n * eps + 16 * eps, r


@pytest.mark.parametrize("n", [256, 257, 319, 320, 321, 513, 700, 768, 769, 1100])
def test_inverse_blocked_gauss_jordan(cuda, n):
    """Blocked Gauss-Jordan inverse (complex64, 256 < n <= 768): ragged last
    blocks, 4 to 12 row blocks (clusters of four) and both sides of its range
    (769, 1100: two or three blocks of the recursion, rows of a larger matrix).
    Every entry takes n rank-one updates on top of ceil(n / 64) block steps;
    condition number below 3: residual below 16 sqrt(n) 2^-24 sqrt(n)."""
    import torch
    A = _dominant(n, 70 + n).astype(np.complex64)
    big = torch.full((n + 1, n), 7.0, dtype=torch.complex64, device="cuda")  # a guard row below
    big[:n] = torch.as_tensor(A, device="cuda")
    scr = torch.empty(int(nat.lib().bem200_inverse_nopiv_workspace_size(nat.C64, n)), dtype=torch.uint8,
                      device="cuda")
    ws = torch.empty(1, dtype=torch.uint8, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.call("bem200_inverse_nopiv", nat.C64, 0, n, nat.ptr(big), n, nat.ptr(ws), 0, nat.ptr(scr), 1e-2,
             nat.ptr(info), nat.stream_ptr())
    assert int(info.item()) == 0
    X = big[:n].cpu().numpy().astype(np.complex128)
    r = np.abs(X @ A.astype(np.complex128) - np.eye(n)).max()
    assert r < 16 * n * 2.0 ** -24, r
    assert bool((big[n] == 7).all())
    # a row exchange needed inside a diagonal block is reported
    B = A.copy()
    B[[130, 170]] = B[[170, 130]]
    big[:n] = torch.as_tensor(B, device="cuda")
    nat.call("bem200_inverse_nopiv", nat.C64, 0, n, nat.ptr(big), n, nat.ptr(ws), 0, nat.ptr(scr), 1e-2,
             nat.ptr(info), nat.stream_ptr())
    assert int(info.item()) == 1


@pytest.mark.parametrize("n,part", [(830, 1.0), (1001, 1.0), (1500, 1.0), (1500, 0.4), (1500, 0.1)])
def test_inverse_in_place_products(cuda, n, part):
    """complex64 inverse whose top products run on the tensor cores in place,
    with the workspace of one pass, one that splits the columns (0.4) and one
    too small to keep the operands (0.1: products through scratch).  The
    operands are rounded to 2^-25 of their row norms: same bound as above."""
    import torch
    A = _dominant(n, 90 + n).astype(np.complex64)
    At = torch.as_tensor(A, device="cuda")
    L = nat.lib()
    scr = torch.empty(int(L.bem200_inverse_nopiv_workspace_size(nat.C64, n)), dtype=torch.uint8, device="cuda")
    wsb = int(part * L.bem200_gemm_workspace_size(1, n, n, n // 2 + 64))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.call("bem200_inverse_nopiv", nat.C64, 1, n, nat.ptr(At), n, nat.ptr(ws), wsb, nat.ptr(scr), 1e-2,
             nat.ptr(info), nat.stream_ptr())
    assert int(info.item()) == 0
    X = At.cpu().numpy().astype(np.complex128)
    r = np.abs(X @ A.astype(np.complex128) - np.eye(n)).max()
    assert r < 16 * n * 2.0 ** -24, r


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 129, 200, 513])
@pytest.mark.parametrize("scale", [0, 500, -500])
def test_pivoted_panel_c128(cuda, n, scale):
    """Partially pivoted complex128 panels (rows rotating through registers):
    ragged last panels, one to several CTAs, ties in the first column (the
    first maximum wins), entries near 2^+-500.  The pivots are scipy's, and
    |P A - L U| <= 8 n eps |L| |U| elementwise, the bound of complex Gaussian
    elimination."""
    import torch
    from scipy.linalg import lu_factor
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A[:, 0] = np.array([1, -1, 1j, -1j])[rng.integers(0, 4, n)]
    A *= 2.0 ** scale
    L = nat.lib()
    At = torch.as_tensor(A, device="cuda").clone()
    rowmap, ipiv = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    wsb = int(L.bem200_getrf_workspace_size(nat.C128, 0, n))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    nat.call("bem200_getrf_ex", nat.C128, 0, n, nat.ptr(At), n, nat.ptr(rowmap), nat.ptr(ipiv), nat.ptr(info),
             nat.ptr(ws), wsb, 0, 0, nat.stream_ptr())
    assert int(info.item()) == 0
    assert np.array_equal(ipiv.cpu().numpy(), lu_factor(A)[1])
    P = rowmap.cpu().numpy()
    F = At.cpu().numpy()[P]
    Lo, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    assert np.all(np.abs(A[P] - Lo @ U) <= 8 * n * 2.0 ** -53 * (np.abs(Lo) @ np.abs(U)))
