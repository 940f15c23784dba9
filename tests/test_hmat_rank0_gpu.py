"""H-matrix operator on a dimer of two metals: G1 and H1 vanish between the
particles (their insides are different regions), so the cross-particle blocks
of these matrices have rank 0.  Against the dense FP64 operator, with the
bound of test_hmat_operator_gpu.py."""
import ctypes

import numpy as np
import pytest

from mnpbem_b200.geometry import ComParticle, trisphere
from mnpbem_b200.materials import EpsConst, EpsDrude
from meshes import DRUDE_AU


def _two_metals():
    a, b = trisphere(144, 10.0), trisphere(144, 10.0)
    a.shift([-6.0, 0, 0])
    b.shift([6.0, 0, 0])
    return ComParticle([EpsConst(1.77), EpsDrude(*DRUDE_AU), EpsDrude(3.7, 9.17, 0.021)], [a, b], [[2, 1], [3, 1]], 1, 2,
                       interp="curv")


def test_two_metals_have_admissible_blocks_between_the_particles():
    from mnpbem_b200.hmatrix import ClusterTree, block_partition, make_kaware_fadmiss, particle_index
    cp = _two_metals()
    tree = ClusterTree(cp.pos, cleaf=33, ipart_arr=particle_index(cp))
    low = np.array(block_partition(tree, make_kaware_fadmiss(2 * np.pi / 620.0))[1])
    assert np.any(tree.ipart[low[:, 0]] != tree.ipart[low[:, 1]])


@pytest.mark.gpu
@pytest.mark.parametrize("fill", ["green", "dense"])
@pytest.mark.parametrize("npol", [1, 2])
def test_operator_with_rank_zero_blocks(cuda, npol, fill):
    import torch
    from mnpbem_b200 import _native as nat
    from mnpbem_b200.bem import BEMRet
    from mnpbem_b200.hmatrix import BEMHMatrices
    cp, enei = _two_metals(), 620.0
    bem = BEMRet(cp)
    bem._eps(enei)
    k, n = 2 * np.pi / enei, cp.n
    gen = torch.Generator(device="cuda").manual_seed(npol)
    x = torch.view_as_complex(torch.randn((8 * n * npol, 2), dtype=torch.float64, device="cuda", generator=gen))
    hm = BEMHMatrices(cp, bem.g, htol=1e-10, kmax=100, cleaf=33).build(enei, fill=fill)
    assert np.any(hm.H[0].ranks == 0) and np.any(hm.H[2].ranks == 0)
    got = torch.empty_like(x)
    hm.apply(npol, bem._eps_mode, bem._e1p, bem._e2p, bem._nvec, k, x, got)
    G = bem.g.bem_matrices(enei)
    scr = torch.empty(int(nat.lib().bem200_bem_apply_workspace_size(n, npol)), dtype=torch.uint8, device="cuda")
    ref = torch.empty_like(x)
    nat.call("bem200_bem_apply", n, npol, *[nat.ptr(m) for m in G], bem._eps_mode, bem._e1p, bem._e2p,
             nat.ptr(bem._nvec), k, nat.ptr(x), ctypes.c_void_p(x.data_ptr() + 16 * 4 * n * npol), None, nat.ptr(ref),
             nat.ptr(scr), nat.stream_ptr())
    assert float((got - ref).abs().max()) <= 1e-8 * float(ref.abs().max())
