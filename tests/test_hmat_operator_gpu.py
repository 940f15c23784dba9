"""bem200_hmat_operator (four H-matrices per launch, row tiles over runs of
blocks) against the dense FP64 operator: compression tolerance 1e-10, so the
products agree to about 1e-10 times the number of blocks in a row; 1e-8 bounds
it.  Small leaf sizes give many blocks per run, a single leaf no low-rank block."""
import ctypes

import numpy as np
import pytest

from meshes import dimer, sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mk,cleaf", [(sphere, 12), (sphere, 40), (sphere, 400), (dimer, 33)],
                         ids=["s12", "s40", "s400", "d33"])
@pytest.mark.parametrize("npol", [1, 2])
def test_hmat_operator_matches_dense(cuda, mk, cleaf, npol):
    import torch
    from mnpbem_b200 import _native as nat
    from mnpbem_b200.bem import BEMRet
    from mnpbem_b200.hmatrix import BEMHMatrices
    cp, enei = mk(), 620.0
    bem = BEMRet(cp)
    bem._eps(enei)
    k = 2 * np.pi / enei
    n = cp.n
    gen = torch.Generator(device="cuda").manual_seed(n + cleaf + npol)
    x = torch.view_as_complex(torch.randn((8 * n * npol, 2), dtype=torch.float64, device="cuda", generator=gen))
    hm = BEMHMatrices(cp, bem.g, htol=1e-10, kmax=100, cleaf=cleaf).build(enei)
    got = torch.empty_like(x)
    hm.apply(npol, bem._eps_mode, bem._e1p, bem._e2p, bem._nvec, k, x, got)
    G = bem.g.bem_matrices(enei)
    scr = torch.empty(int(nat.lib().bem200_bem_apply_workspace_size(n, npol)), dtype=torch.uint8, device="cuda")
    ref = torch.empty_like(x)
    nat.call("bem200_bem_apply", n, npol, *[nat.ptr(m) for m in G], bem._eps_mode, bem._e1p, bem._e2p,
             nat.ptr(bem._nvec), k, nat.ptr(x), ctypes.c_void_p(x.data_ptr() + 16 * 4 * n * npol), None, nat.ptr(ref),
             nat.ptr(scr), nat.stream_ptr())
    assert float((got - ref).abs().max()) <= 1e-8 * float(ref.abs().max())
