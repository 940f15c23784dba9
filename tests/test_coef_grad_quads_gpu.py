"""Vertex gradient on quadrilateral faces: the reverse-mode derivatives of the
refinement quadrature on curved quads (nine nodes for the self term, two
six-node triangles for near pairs) against central differences of the solver,
with the tolerance of test_vertex_grad_gpu.py (same step, same noise)."""
import numpy as np
import pytest

from test_vertex_grad_gpu import _bem, _fd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [6, 9])
def test_vertex_gradient_of_quad_faces(cuda, m):
    from mnpbem_b200 import ComParticle, EpsConst, EpsDrude, PlaneWaveRet
    from mnpbem_b200.geometry import tricube
    from mnpbem_b200.shape import extinction_vertex_vjp, random_directions
    cp = ComParticle([EpsConst(1.0), EpsDrude(9.84, 9.0, 0.067)], [tricube(m, 40.0, 0.25, interp="curv")], [[2, 1]], 1,
                     interp="curv")
    pol, dirs, enei = np.array([[1.0, 0, 0]]), np.array([[0, 0, 1.0]]), 580.0
    ext, grad = extinction_vertex_vjp(_bem(cp, enei, "fp64"), PlaneWaveRet(pol, dirs), enei)
    assert np.all(np.abs(grad.sum(axis=0)) <= 1e-9 * np.abs(grad).sum(axis=0)), grad.sum(axis=0)
    for D in random_directions(cp, 2, seed=3):
        ref = float(_fd(cp, D, enei, pol, dirs)[0])
        got = float(np.sum(grad * D))
        assert abs(got - ref) <= 2e-6 * max(abs(ref), 1e-3 * np.max(np.abs(ext))), (got, ref)
