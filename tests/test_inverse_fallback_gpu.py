"""A mixed solve whose explicit inverses turn out too inaccurate (their probe is
coarse) is repeated with LU factors instead of failing.  The bad inverse is made
here by overwriting G1^-1 in the workspace."""

import numpy as np
import pytest

from meshes import sphere

pytestmark = pytest.mark.gpu

POL, DIR = np.array([[1.0, 0, 0]]), np.array([[0, 0, 1.0]])


def _bad_inverses(**kw):
    from mnpbem_b200 import BEMRet
    cp = sphere()
    bem = BEMRet(cp, precision="mixed", gmres_maxit=5, **kw)
    bem.init(600.0)
    assert bem.last_pivoting == "inverse"
    off = bem._slots[0] - bem._ws.data_ptr()
    bem._ws[off:off + 8 * cp.n * cp.n].zero_()
    return cp, bem


@pytest.mark.parametrize("gmres_ir", [True, False])
def test_solve_falls_back_to_lu(cuda, gmres_ir):
    from mnpbem_b200 import BEMRet, PlaneWaveRet
    cp, bem = _bad_inverses(gmres_ir=gmres_ir)
    exc = PlaneWaveRet(POL, DIR)
    ref = exc.extinction(BEMRet(cp).solve(exc.potential(cp, 600.0))[0])
    sig, _ = bem.solve(exc.potential(cp, 600.0))
    assert bem.last_pivoting in ("diagonal", "partial")
    assert abs(exc.extinction(sig) - ref) <= 1e-10 * abs(ref)
    bem.clear()  # the next wavelength tries the inverses again
    bem.solve(exc.potential(cp, 610.0))
    assert bem.last_pivoting == "inverse"


def test_transposed_solve_falls_back_to_lu(cuda):
    import torch
    from mnpbem_b200 import BEMRet
    from mnpbem_b200.shape import _transposed_solve
    cp, bem = _bad_inverses()
    w = torch.randn(8 * cp.n, dtype=torch.complex128, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    lam, _ = _transposed_solve(bem, w, 1)
    assert bem.last_pivoting in ("diagonal", "partial")
    ref, _ = _transposed_solve(BEMRet(cp, enei=600.0), w, 1)
    assert float((lam - ref).abs().max()) <= 1e-9 * float(ref.abs().max())
