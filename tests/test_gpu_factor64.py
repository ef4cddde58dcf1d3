"""The complex128 LDL^T at the edges of its tiles (64), middle panels (256) and
block columns (1,024), with its updates on the INT8 tensor cores and on the
FP64 pipe, and with pivots outside the range of the fast reciprocal."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = 2 * math.pi / 0.1


def _device(nx, ny, eta0=376.730313668):
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.005 * nx, 0.005 * ny, nx, ny)
    dev = EFIEDevice(mesh, build_rwg(mesh))
    Z = dev.assemble(K, eta0=eta0, copy_out=True)
    return dev, Z


def _backward_error(dev, Z, tensor_cores):
    dev.set_option("tensor_cores", tensor_cores)
    dev.build_nearfield(math.inf, "lu")
    rng = np.random.default_rng(3)
    b = rng.standard_normal(dev.N) + 1j * rng.standard_normal(dev.N)
    x = dev.nf_apply(b)
    return np.linalg.norm(Z @ x - b) / (np.linalg.norm(Z) * np.linalg.norm(x))


# N = 3 nx ny - nx - ny: one ragged tile, tile and panel edges with their
# remainders, one and two block columns (the K = 1,024 update), 2,640
@pytest.mark.parametrize("nx,ny", [(3, 4), (4, 6), (5, 5), (9, 10), (9, 11), (13, 14), (18, 20), (21, 21), (20, 23),
                                   (30, 30)])
@pytest.mark.parametrize("tensor_cores", [1, 0])
def test_backward_error(nx, ny, tensor_cores):
    dev, Z = _device(nx, ny)
    # each entry of the factor carries a sum of up to N products: the error
    # bound of an FP64 sum is N 2^-53 of its magnitudes (twice: L D L^T and the
    # two sweeps)
    assert _backward_error(dev, Z, tensor_cores) < dev.N * 2.0 ** -52
    dev.close()


def test_int8_update_no_worse_than_fp64_pipe():
    """On a two-block-column matrix the int8 residue updates leave no larger an
    error than the FP64 pipe's sums (both are rounding: a factor of two covers
    their scatter)."""
    dev, Z = _device(30, 30)
    e8, e64 = _backward_error(dev, Z, 1), _backward_error(dev, Z, 0)
    dev.close()
    assert e8 < 2 * e64


def _graded_plate(power):
    from diffmom_b200 import TriMesh, make_rect_plate
    m = make_rect_plate(0.06, 0.06, 18, 20)
    xyz = m.xyz.copy()
    lo = xyz[:, 0].min()
    xyz[:, 0] = lo + 0.06 * ((xyz[:, 0] - lo) / 0.06) ** power
    return TriMesh(xyz, m.tri)


@pytest.mark.parametrize("mesh", ["disk", "graded 4", "graded 7"])
def test_int8_update_on_graded_meshes(mesh):
    """Slivers and cells graded over decades: basis functions of scales up to
    3e6 apart.  The residual is compared row by row with |Z| |x|, so that rows
    of small scale count as the others do."""
    from diffmom_b200 import EFIEDevice, build_rwg, make_circular_plate
    mesh = make_circular_plate(0.05, 12, 48) if mesh == "disk" else _graded_plate(int(mesh.split()[1]))
    dev = EFIEDevice(mesh, build_rwg(mesh))
    Z = dev.assemble(K, copy_out=True)
    rng = np.random.default_rng(3)
    b = (rng.standard_normal(dev.N) + 1j * rng.standard_normal(dev.N)) * np.sqrt(np.abs(np.diag(Z)))
    omega = {}
    for tensor_cores in (1, 0):
        dev.set_option("tensor_cores", tensor_cores)
        dev.build_nearfield(math.inf, "lu")
        x = dev.nf_apply(b)
        r = Z.astype(np.clongdouble) @ x.astype(np.clongdouble) - b
        omega[tensor_cores] = float(np.max(np.abs(r) / (np.abs(Z) @ np.abs(x))))
    dev.close()
    # both are rounding, seen through the growth of an elimination without
    # pivoting: a factor of four covers the scatter of a largest row
    assert omega[1] < 4 * omega[0], omega


def test_pivots_outside_the_fast_range():
    """|pivot|^2 underflows; the factor does not (the matrix is scaled by a
    power of two, which changes no rounding of a sum)."""
    scale = 2.0 ** -560
    dev, Z = _device(13, 14, eta0=376.730313668 * scale)
    dev.build_nearfield(math.inf, "lu")
    b = np.random.default_rng(5).standard_normal(dev.N) + 0j
    x = dev.nf_apply(b * scale)
    Zs = Z / scale
    dev.close()
    assert np.linalg.norm(Zs @ x - b) / (np.linalg.norm(Zs) * np.linalg.norm(x)) < dev.N * 2.0 ** -52
