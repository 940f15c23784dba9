"""Engine 0 means FP64 products on the CUDA cores for complex128 whatever the
workspace, in the LU and in the init of the dense solver; engine 1 takes the
tensor cores when their operand space is given."""
import ctypes

import numpy as np
import pytest

from mnpbem_b200 import _native as nat


def test_operand_space_belongs_to_engine_1():
    L = nat.lib()
    n = 1537
    assert L.bem200_getrf_workspace_size(nat.C128, 0, n) < (1 << 20)
    assert L.bem200_getrf_workspace_size(nat.C128, 1, n) > (64 << 20)
    # seven matrices, pivots, LU scratch and diagonal-block inverses: no operand space
    assert L.bem200_bem_workspace_size(0, n) < 16 * 7 * n * n + 16 * 6 * 64 * (n + 64) + (2 << 20)
    assert L.bem200_bem_gemm_workspace_size(0, 0, n) == 0
    assert L.bem200_bem_gemm_workspace_size(0, 1, n) > (64 << 20)
    assert L.bem200_bem_gemm_workspace_size(1, 1, n) == 2 * L.bem200_gemm_workspace_size(1, n, n, n)
    assert L.bem200_bem_gemm_workspace_size(0, 1, 0) == 0


def _dominant(n, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g)
    return A / n ** 0.5 + 4 * torch.eye(n, dtype=A.dtype, device="cuda")


def _getrf(A, engine, wsb, flags):
    import torch
    n = A.shape[0]
    F = A.clone()
    rowmap, ipiv = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    nat.call("bem200_getrf_ex", nat.C128, engine, n, nat.ptr(F), n, nat.ptr(rowmap), nat.ptr(ipiv), nat.ptr(info),
             nat.ptr(ws), wsb, flags, 0, nat.stream_ptr())
    assert int(info.item()) == 0
    return F


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [0, 4])
def test_getrf_engine_0_ignores_the_workspace_size(cuda, flags):
    import torch
    n = 1100
    L = nat.lib()
    A = _dominant(n, 3)
    small, big = (int(L.bem200_getrf_workspace_size(nat.C128, e, n)) for e in (0, 1))
    ref = _getrf(A, 0, small, flags)
    assert torch.equal(ref, _getrf(A, 0, big, flags))
    assert torch.equal(ref, _getrf(A, 1, small, flags))       # no room for operands
    tc = _getrf(A, 1, big, flags)
    assert not torch.equal(ref, tc) and float((ref - tc).abs().max()) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("engine", [0, 1])
def test_init_factors_on_the_chosen_engine(cuda, engine):
    """LU(G1) of a precision 0 init is bem200_getrf's on the same engine."""
    import torch
    L = nat.lib()
    n = 1100
    ws = torch.empty(int(L.bem200_bem_workspace_size(0, n)), dtype=torch.uint8, device="cuda")
    slots = [ctypes.c_void_p() for _ in range(4)]
    nat.call("bem200_bem_slots", 0, n, nat.ptr(ws), *[ctypes.byref(s) for s in slots])

    def slot(i):
        off = slots[i].value - ws.data_ptr()
        return ws[off:off + 16 * n * n].view(torch.complex128).view(n, n)
    mats = [_dominant(n, 10 + i) for i in range(4)]
    mats[3] = -mats[3]
    for i, m in enumerate(mats):
        slot(i).copy_(m)
    nvec = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    nvec[:, 2] = 1
    e1, e2 = (ctypes.c_double * 2)(-11.0, 1.2), (ctypes.c_double * 2)(1.77, 0.0)
    gb = int(L.bem200_bem_gemm_workspace_size(0, 1, n))  # given to engine 0 as well
    gws = torch.empty(gb, dtype=torch.uint8, device="cuda")
    info = ctypes.c_int32(0)
    nat.call("bem200_bem_init", 0, engine, n, nat.ptr(ws), 0, ctypes.cast(e1, ctypes.c_void_p),
             ctypes.cast(e2, ctypes.c_void_p), nat.ptr(nvec), 0.01, nat.ptr(gws), gb, ctypes.byref(info), nat.stream_ptr())
    ref = [_getrf(mats[0], e, int(L.bem200_getrf_workspace_size(nat.C128, e, n)), 0) for e in (0, 1)]
    assert not torch.equal(ref[0], ref[1])
    assert torch.equal(slot(0), ref[engine])


@pytest.mark.gpu
def test_fp64_solver_engines_agree(cuda):
    from meshes import rel, sphere
    from mnpbem_b200 import PlaneWaveRet
    from mnpbem_b200.bem import BEMRet
    cp = sphere(484)
    exc = PlaneWaveRet(np.array([[1.0, 0, 0]]), np.array([[0, 0, 1.0]]))
    out = []
    for engine in ("simt", "bf16x3"):
        bem = BEMRet(cp, precision="fp64", engine=engine)
        sig, _ = bem.solve(exc.potential(cp, 600.0))
        assert bem.engine == engine
        out.append((sig.sig1, sig.h2, np.asarray(exc.extinction(sig))))
    for a, b in zip(*out):
        assert rel(a, b) < 1e-9
