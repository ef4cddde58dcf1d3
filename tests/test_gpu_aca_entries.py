"""Entries of the H-matrix operator, formed from quadrature data laid out in
tree order with one shared row or column in shared memory, against the dense
FP64 Z: every quadrature order, ragged leaf sizes, blocks of arbitrary index
lists and ranks beyond those whose factors are kept in shared memory (64)."""
import math

import numpy as np
import pytest

from diffmom_b200 import (EFIEDevice, RWGData, TriMesh, aca_lowrank, build_aca_operator, build_efie_cache, build_rwg,
                          make_rect_plate)

pytestmark = pytest.mark.gpu

K = 2 * math.pi / 0.1
EPS = np.finfo(float).eps


def _plate(nx, ny, quad_order):
    m = make_rect_plate(0.1, 0.12, nx, ny)
    r = build_rwg(m)
    dev = EFIEDevice(m, r)
    Z = dev.assemble(K, quad_order=quad_order, precision="fp64", copy_out=True)
    dev.close()
    return m, r, Z


def _bound(Z, quad_order):
    # an entry sums 4 nq^2 products, whose vector and charge parts cancel to
    # about a tenth; each carries some 30 rounding errors
    return (4 * quad_order ** 2 + 30) * 10 * EPS * np.abs(Z).max()


@pytest.mark.parametrize("quad_order", [1, 3, 4, 7])
@pytest.mark.parametrize("leaf_size", [1, 7, 33])
def test_dense_blocks_and_entries(quad_order, leaf_size):
    m, r, Z = _plate(5, 7, quad_order)
    A = build_aca_operator(m, r, K, leaf_size=leaf_size, aca_tol=1e-10, quad_order=quad_order)
    p = A.perm - 1
    for b in A.dense_blocks:
        rows, cols = p[b.row_range.start - 1:b.row_range.stop - 1], p[b.col_range.start - 1:b.col_range.stop - 1]
        assert np.abs(b.data - Z[np.ix_(rows, cols)]).max() <= _bound(Z, quad_order)
    n = r.nedges
    i, j = np.divmod(np.arange(n * n), n)
    E = A.entries(i + 1, j + 1).reshape(n, n)
    assert np.abs(E - Z).max() <= _bound(Z, quad_order)
    A.close()


@pytest.mark.parametrize("m_rows,n_cols", [(1, 1), (3, 70), (90, 75), (130, 66)])
def test_lowrank_of_index_lists(m_rows, n_cols):
    # all pivots taken: the cross approximation is the block itself, up to the
    # growth of the elimination (bounded here by the square of the rank)
    m, r, Z = _plate(9, 9, 3)
    rng = np.random.default_rng(m_rows)
    rows, cols = rng.permutation(r.nedges)[:m_rows], rng.permutation(r.nedges)[:n_cols]
    cache = build_efie_cache(m, r, K, quad_order=3)
    q = min(m_rows, n_cols)
    U, V = aca_lowrank(cache, rows + 1, cols + 1, tol=1e-15, max_rank=q)
    S = Z[np.ix_(rows, cols)]
    assert U.shape[1] == V.shape[1] <= q
    assert np.linalg.norm(U @ V.conj().T - S) <= 100 * (q * q + 30) * EPS * np.linalg.norm(S)


def test_neighbours_without_a_common_basis_function():
    """Two slender triangles with a common edge that carries no basis function;
    all slots of each belong to another edge, where three triangles are
    attached.  Their entries take the near terms as the dense matrix does."""
    L, e = 0.01, 0.001
    v1, v2, v3, w = [-L, 3 * e, 0], [0, e, 0], [0, -e, 0], [L, -3 * e, 0]
    tips = [[x, 0, z] for x in (-L / 2, L / 2) for z in (0.004, -0.005, 0.007)]
    xyz = np.array([v1, v2, v3, w] + tips)
    tri = np.array([[1, 2, 3], [4, 3, 2]] + [[1, 3, 5 + i] for i in range(3)] + [[4, 2, 8 + i] for i in range(3)])
    mesh = TriMesh(xyz, tri)
    one, edge = np.repeat([1, 2], 3), np.repeat([[1, 3], [2, 4]], 3, axis=0)
    length = np.linalg.norm(xyz[edge[:, 0] - 1] - xyz[edge[:, 1] - 1], axis=1)
    T = xyz[tri - 1]
    area = 0.5 * np.linalg.norm(np.cross(T[:, 1] - T[:, 0], T[:, 2] - T[:, 0]), axis=1)
    tminus = np.arange(3, 9)
    rwg = RWGData(mesh=mesh, nedges=6, tplus=one, tminus=tminus, evert=edge, vplus_opp=np.repeat([2, 3], 3),
                  vminus_opp=np.arange(5, 11), len=length, area_plus=area[one - 1], area_minus=area[tminus - 1],
                  coeff_plus=np.ones(6), coeff_minus=np.ones(6))
    dev = EFIEDevice(mesh, rwg)
    Z = dev.assemble(K, copy_out=True)
    dev.close()
    A = build_aca_operator(mesh, rwg, K)
    i, j = np.divmod(np.arange(36), 6)
    E = A.entries(i + 1, j + 1).reshape(6, 6)
    A.close()
    assert np.abs(E - Z).max() <= _bound(Z, 3)
