"""The FP64 matrix-instruction GEMM at the edges of its 32 x 64 tiles and 16-deep
chunks: Z X with many columns, many-column sweeps (plain and transposed factor)
and the factor's trailing updates without the tensor cores."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# N = 3 nx ny - nx - ny: 1, 29, 33, 280, 1,042
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 4), (2, 7), (10, 10), (18, 20)])
@pytest.mark.parametrize("columns", [16, 63, 64, 65, 130])
def test_products_and_sweeps(nx, ny, columns):
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.005 * nx, 0.005 * ny, nx, ny)
    dev = EFIEDevice(mesh, build_rwg(mesh))
    Z = dev.assemble(2 * math.pi / 0.1, precision="fp64", copy_out=True)
    dev.set_option("tensor_cores", 0)
    dev.build_nearfield(math.inf, "lu")
    rng = np.random.default_rng(columns)
    B = np.asfortranarray(rng.standard_normal((dev.N, columns)) + 1j * rng.standard_normal((dev.N, columns)))
    Y, X = dev.matvec(B), dev.nf_apply(B)
    dev.close()
    # N products of four terms in FP64: N 2^-52 of the magnitudes
    tol = dev.N * 2.0 ** -51
    assert np.all(np.abs(Y - Z @ B) <= tol * (np.abs(Z) @ np.abs(B)))
    for r in range(columns):
        assert np.linalg.norm(Z @ X[:, r] - B[:, r]) < tol * np.linalg.norm(Z) * np.linalg.norm(X[:, r])
