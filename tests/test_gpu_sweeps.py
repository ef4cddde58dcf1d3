"""The few-column triangular sweeps at the edges of their 16-row slices and
256-row blocks, one to seven columns, complex128 and complex64 factors."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# N = 3 nx ny - nx - ny: 5, 16, 29, 208, 251, 280, 527, 1042
@pytest.mark.parametrize("nx,ny", [(1, 3), (2, 4), (3, 4), (8, 10), (9, 10), (10, 10), (13, 15), (18, 20)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sweeps_solve(nx, ny, precision):
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.005 * nx, 0.005 * ny, nx, ny)
    dev = EFIEDevice(mesh, build_rwg(mesh))
    Z = dev.assemble(2 * math.pi / 0.1, precision=precision, copy_out=True)
    dev.build_nearfield(math.inf, "lu")
    rng = np.random.default_rng(nx)
    B = rng.standard_normal((dev.N, 7)) + 1j * rng.standard_normal((dev.N, 7))
    one = dev.nf_apply(B[:, 0])
    many = dev.nf_apply(np.asfortranarray(B))
    dev.close()
    # the factor's own rounding: N sums of its precision (see the backward
    # error bound of an FP64 or FP32 factorisation)
    tol = dev.N * (2.0 ** -52 if precision == "fp64" else 2.0 ** -23)
    for r in range(7):
        res = np.linalg.norm(Z @ many[:, r] - B[:, r])
        assert res < tol * np.linalg.norm(Z) * np.linalg.norm(many[:, r])
    assert np.array_equal(one, many[:, 0])  # a column's sums do not depend on the others


def test_new_factor_between_solves():
    """Solves whose iterations are replayed graphs follow a new factor."""
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.1, 0.1, 12, 12)
    dev = EFIEDevice(mesh, build_rwg(mesh))
    rng = np.random.default_rng(1)
    b = rng.standard_normal(dev.N) + 1j * rng.standard_normal(dev.N)
    for k in (60.0, 60.0, 75.0, 90.0):
        for repeat in range(3):
            if repeat == 0:
                Z = dev.assemble(k, copy_out=True)
                P = dev.build_nearfield(math.inf, "lu")
            x, st = dev.gmres(b, tol=1e-10, maxiter=20, preconditioner=P, precond_side="right")
            assert st.niter <= 2
            assert np.linalg.norm(Z @ x - b) < 1e-9 * np.linalg.norm(b)
    dev.close()


def test_nan_with_the_empty_pattern():
    """A NaN of all ones in the right-hand side, the pattern of a value not yet
    there, passes through as a NaN; the next solve is right."""
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.05, 0.05, 12, 12)
    dev = EFIEDevice(mesh, build_rwg(mesh))
    Z = dev.assemble(2 * math.pi / 0.1, precision="fp64", copy_out=True)
    dev.build_nearfield(math.inf, "lu")
    b = np.ones(dev.N, dtype=np.complex128)
    bad = b.copy()
    bad.view(np.uint64)[6:8] = 0xffffffffffffffff
    assert np.isnan(dev.nf_apply(bad)).any()
    x = dev.nf_apply(b)
    dev.close()
    assert np.linalg.norm(Z @ x - b) < dev.N * 2.0 ** -52 * np.linalg.norm(Z) * np.linalg.norm(x)


def test_many_contexts_sweep_at_once():
    """Twenty contexts of seven columns: more waiting CTAs than the GPU holds."""
    from concurrent.futures import ThreadPoolExecutor
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.09, 0.1, 18, 20)
    rwg = build_rwg(mesh)
    rng = np.random.default_rng(2)
    B = np.asfortranarray(rng.standard_normal((rwg.nedges, 7)) + 1j * rng.standard_normal((rwg.nedges, 7)))
    devs = [EFIEDevice(mesh, rwg) for _ in range(20)]
    for dev in devs:
        dev.assemble(2 * math.pi / 0.1)
        dev.build_nearfield(math.inf, "lu")
    alone = devs[0].nf_apply(B)
    with ThreadPoolExecutor(len(devs)) as pool:
        for X in pool.map(lambda dev: [dev.nf_apply(B) for _ in range(10)], devs):
            for x in X:
                np.testing.assert_array_equal(x, alone)
    for dev in devs:
        dev.close()
