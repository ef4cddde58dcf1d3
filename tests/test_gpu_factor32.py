"""The complex64 LDL^T at the edges of its 16 x 16 blocks, tiles (64), middle
panels (256) and block columns (1,024), with its updates on the tensor cores and
on FP32 units."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = 2 * math.pi / 0.1


# N = 3 nx ny - nx - ny
@pytest.mark.parametrize("nx,ny", [(2, 3), (3, 4), (4, 6), (5, 5), (9, 10), (9, 11), (13, 14), (18, 20), (21, 21),
                                   (20, 23), (30, 30)])
@pytest.mark.parametrize("tensor_cores", [1, 0])
def test_backward_error(nx, ny, tensor_cores):
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.005 * nx, 0.005 * ny, nx, ny)
    dev = EFIEDevice(mesh, build_rwg(mesh))
    Z = dev.assemble(K, precision="mixed", copy_out=True)
    dev.set_option("tensor_cores", tensor_cores)
    dev.build_nearfield(math.inf, "lu")
    rng = np.random.default_rng(3)
    b = rng.standard_normal(dev.N) + 1j * rng.standard_normal(dev.N)
    x = dev.nf_apply(b)
    dev.close()
    # each entry of the factor carries a sum of up to N products: the error
    # bound of an FP32 sum is N 2^-24 of its magnitudes (twice: L D L^T and the
    # two sweeps)
    assert np.linalg.norm(Z @ x - b) < dev.N * 2.0 ** -23 * np.linalg.norm(Z) * np.linalg.norm(x)
