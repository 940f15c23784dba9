"""The block partition one level at a time (admissibility rules with an array form)
against the recursion over pairs, which custom rules still take: the same blocks
in the same order."""
import numpy as np
import pytest

from mnpbem_b200 import hmatrix as hm
import meshes


def _two_sizes():
    from mnpbem_b200.geometry import ComParticle, trisphere
    from mnpbem_b200.materials import EpsConst, EpsDrude
    a, b = trisphere(144, 10.0), trisphere(60, 4.0)
    b.shift([9.0, 1.0, 0.5])
    return ComParticle([EpsConst(1.77), EpsDrude(*meshes.DRUDE_AU)], [a, b], [[2, 1], [2, 1]], 1, 2, interp="curv")


@pytest.mark.parametrize("mk", [lambda: meshes.sphere(324), meshes.dimer, _two_sizes,
                                lambda: meshes.shape_particle("rodbem"), lambda: meshes.shape_particle("cubebem")],
                         ids=["sphere", "dimer", "two_sizes", "rod", "cube"])
@pytest.mark.parametrize("cleaf", [1, 8, 33, 2000])
def test_array_form_equals_recursion(mk, cleaf):
    cp = mk()
    tree = hm.ClusterTree(cp.pos, cleaf=cleaf, ipart_arr=hm.particle_index(cp))
    for k in (2 * np.pi / 620.0, 0.3, 3.0 + 1.0j):
        rule = hm.make_kaware_fadmiss(k)
        assert hasattr(rule, "many")
        ref = hm.block_partition(tree, lambda r1, r2, d: rule(r1, r2, d))
        got = hm.block_partition(tree, rule)
        for a, b in zip(got, ref):
            assert a == [tuple(int(i) for i in v) for v in b]


@pytest.mark.parametrize("cleaf,kmax", [(1, 4), (8, 100), (33, 100), (2000, 100)])
def test_work_items_cover_every_block(cleaf, kmax):
    """Items of the products: 128 rows of V, 32 rows of a block, and the operator's
    tiles, which hold every row of every block once and at most 128 blocks."""
    cp = _two_sizes()
    tree = hm.ClusterTree(cp.pos, cleaf=cleaf, ipart_arr=hm.particle_index(cp))
    dense, low = hm.block_partition(tree, hm.make_kaware_fadmiss(2 * np.pi / 620.0))
    L = hm._Layout(tree, dense, low, kmax, "cpu")
    nd = len(L.db)
    assert [tuple(v) for v in L.db] == [(tree.cind[a, 0], tree.cind[a, 1] - tree.cind[a, 0] + 1, tree.cind[b, 0],
                                         tree.cind[b, 1] - tree.cind[b, 0] + 1) for a, b in dense]
    vit = [(l, j) for l in range(len(L.lb)) for j in range(0, int(L.lb[l, 3]), 128)]
    bit = [(b, i) for b in range(nd) for i in range(0, int(L.db[b, 1]), 32)]
    bit += [(nd + l, i) for l in range(len(L.lb)) for i in range(0, int(L.lb[l, 1]), 32)]
    assert [tuple(v) for v in L.dev["vitems"].numpy().reshape(-1, 2)] == vit
    assert [tuple(v) for v in L.dev["bitems"].numpy().reshape(-1, 2)] == bit
    blocks = np.concatenate([L.db, L.lb])
    seen = np.zeros((len(blocks), cp.n), dtype=int)
    lst = L.dev["blist"].numpy()
    for row, nrow, lo, hi in L.dev["tiles"].numpy().reshape(-1, 4):
        assert 0 < nrow <= 32 and 0 < hi - lo <= 128
        seen[lst[lo:hi], row:row + nrow] += 1
    for b, (r0, m, _, _) in enumerate(blocks):
        assert np.all(seen[b, r0:r0 + m] == 1) and seen[b].sum() == m
