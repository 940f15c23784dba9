"""A fill of the four H-matrices that fails leaves nothing running on memory that
the caller's stream may get: the fills already queued on side streams are joined
into it."""
import pytest

from meshes import sphere

pytestmark = pytest.mark.gpu


def test_failing_fill_is_joined(cuda, monkeypatch):
    import torch
    from mnpbem_b200.bem import BEMRet
    from mnpbem_b200.hmatrix import BEMHMatrices, HMatrixGPU
    cp = sphere()
    bem = BEMRet(cp)
    hm = BEMHMatrices(cp, bem.g, htol=1e-8, kmax=100, cleaf=32)
    load, done = torch.randn((3000, 3000), dtype=torch.float64, device="cuda"), torch.cuda.Event()
    torch.cuda.synchronize()

    def fill(self, g, enei, which, fetch=True):
        if which == 2:
            raise MemoryError("third fill")
        for _ in range(20):
            load @ load
        done.record()
    with monkeypatch.context() as m:
        m.setattr(HMatrixGPU, "compress_green", fill)
        with pytest.raises(MemoryError):
            hm.build(620.0)
    assert hm.H is None
    torch.cuda.current_stream().synchronize()
    assert done.query()
    hm.build(620.0)  # and the object is good for another try
    assert len(hm.H) == 4 and all(h.ranks is not None for h in hm.H)
