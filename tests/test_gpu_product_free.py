"""The matrix-free product against the dense matrix at the edges of its tiles
(128 test triangles a CTA, 32 source triangles a tile, chunks), every
quadrature order, and an edge shared by three triangles."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(mesh, quad_order):
    from diffmom_b200 import EFIEDevice, build_rwg, matrixfree_efie_operator
    rwg = build_rwg(mesh)
    k = 2 * math.pi / 0.1
    dev = EFIEDevice(mesh, rwg)
    Z = dev.assemble(k, quad_order=quad_order, copy_out=True)
    dev.close()
    rng = np.random.default_rng(quad_order)
    x = rng.standard_normal(rwg.nedges) + 1j * rng.standard_normal(rwg.nedges)
    y = matrixfree_efie_operator(mesh, rwg, k, quad_order=quad_order) @ x
    # N-term FP64 sums in another order; entries carry a few roundings of the
    # kernel each
    assert np.linalg.norm(y - Z @ x) < 1e-13 * np.linalg.norm(Z) * np.linalg.norm(x)


@pytest.mark.parametrize("quad_order", [1, 3, 4, 7])
@pytest.mark.parametrize("nx,ny", [(2, 2), (4, 4), (5, 13), (8, 8), (9, 15)])
def test_matrix_free_matches_dense(nx, ny, quad_order):
    from diffmom_b200 import make_rect_plate
    _check(make_rect_plate(0.01 * nx, 0.01 * ny, nx, ny), quad_order)


# chunks of 4, of an odd size between, and of a whole tile (4, 392 and 1,250 triangles)
@pytest.mark.parametrize("quad_order", [1, 7])
@pytest.mark.parametrize("nx,ny", [(1, 2), (14, 14), (25, 25)])
def test_matrix_free_chunks(nx, ny, quad_order):
    from diffmom_b200 import make_rect_plate
    _check(make_rect_plate(0.01 * nx, 0.01 * ny, nx, ny), quad_order)


def test_matrix_free_junction():
    from diffmom_b200 import TriMesh, make_rect_plate
    m = make_rect_plate(0.1, 0.1, 4, 4)
    # a fin standing on two edges of the plate's middle line: triangles with
    # more than three edge neighbours
    mid = [i + 1 for i in range(m.nvertices) if abs(m.xyz[i, 1]) < 1e-12][:3]
    top = m.xyz[[v - 1 for v in mid]] + np.array([0.0, 0.0, 0.02])
    n = m.nvertices
    tri = [[mid[0], mid[1], n + 1], [mid[1], n + 2, n + 1], [mid[1], mid[2], n + 2], [mid[2], n + 3, n + 2]]
    _check(TriMesh(np.vstack([m.xyz, top]), np.vstack([m.tri, tri])), 3)
