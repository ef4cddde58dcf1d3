"""Results around the size from which copies to the host are staged in chunks
(2 MB, chunks of 1 MB), and contexts that solve repeatedly without growing."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# N^2 x 16 bytes: 1.9 and 2.2 MB (below and above the limit), 17.4 MB (a ragged
# last chunk)
@pytest.mark.parametrize("nx,ny", [(10, 13), (11, 12), (18, 20)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_matrix_copy_equals_entries(nx, ny, precision):
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.005 * nx, 0.005 * ny, nx, ny)
    dev = EFIEDevice(mesh, build_rwg(mesh))
    Z = dev.assemble(2 * math.pi / 0.1, precision=precision, copy_out=True)
    rng = np.random.default_rng(0)
    m = np.concatenate([rng.integers(1, dev.N + 1, 4000), [1, dev.N, dev.N]])
    n = np.concatenate([rng.integers(1, dev.N + 1, 4000), [1, 1, dev.N]])
    assert np.array_equal(Z[m - 1, n - 1], dev.entries(m, n))
    X = rng.standard_normal((dev.N, 300)) + 1j * rng.standard_normal((dev.N, 300))
    Y = dev.matvec(np.asfortranarray(X))
    assert np.linalg.norm(Y - Z @ X) < 1e-11 * np.linalg.norm(Z) * np.linalg.norm(X)
    dev.close()


def test_repeated_calls_keep_device_memory():
    import torch
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.1, 0.1, 24, 24)
    rwg = build_rwg(mesh)
    dev = EFIEDevice(mesh, rwg)
    k = 2 * math.pi / 0.1
    b = np.ones(rwg.nedges, dtype=complex)
    d = np.random.default_rng(0).standard_normal((400, 3))

    def calls():
        dev.assemble(k, copy_out=True)
        P = dev.build_nearfield(0.05, "lu")
        x, _ = dev.gmres(b, tol=1e-8, preconditioner=P)
        dev.solve_direct(b)
        dev.matvec(np.asfortranarray(np.stack([b] * 50, 1)))
        dev.farfield(d, x)
        dev.plane_wave_rhs([[0, 0, -k]], [1.0], [[1, 0, 0]])

    calls()
    calls()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(20):
        calls()
    # one pass takes over 100 MB of buffers: any of them allocated again would show
    assert free - torch.cuda.mem_get_info()[0] < 32 << 20
    dev.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pinned_destination(precision):
    """A pinned destination takes the matrix at the bus rate: faster than the
    staged copy into pageable memory, and the same values."""
    import time
    import torch
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    from diffmom_b200 import _native as nat
    mesh = make_rect_plate(0.125, 0.125, 25, 25)  # 53 MB
    dev = EFIEDevice(mesh, build_rwg(mesh))
    code = nat.PREC_FP64 if precision == "fp64" else nat.PREC_MIXED
    pinned = torch.empty((dev.N, dev.N), dtype=torch.complex128).pin_memory().numpy()
    seconds = {}
    for name, Z in (("pinned", pinned), ("pageable", np.empty((dev.N, dev.N), dtype=np.complex128))):
        times = []
        for _ in range(8):
            Z[:] = 0
            t = time.perf_counter()
            dev.ctx.call("dmb_assemble_z", 2 * math.pi / 0.1, 376.730313668, 3, code, nat.dptr(Z))
            times.append(time.perf_counter() - t)
        seconds[name] = min(times)
        np.testing.assert_array_equal(Z, dev.assemble(2 * math.pi / 0.1, precision=precision, copy_out=True))
    dev.close()
    print(seconds)
    assert seconds["pinned"] < seconds["pageable"]


def test_contexts_share_the_chunks():
    """Large results of many contexts, one after another and from several
    threads at once: the chunks are the device's, so a context's first result
    neither makes its own nor keeps device memory for them."""
    from concurrent.futures import ThreadPoolExecutor
    import torch
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.06, 0.06, 18, 20)  # 17.4 MB
    rwg = build_rwg(mesh)
    k = 2 * math.pi / 0.1
    devs = [EFIEDevice(mesh, rwg) for _ in range(12)]
    for dev in devs:
        dev.assemble(k)
    ref = [devs[0].assemble(k, copy_out=True) for _ in range(4)][-1]
    free = torch.cuda.mem_get_info()[0]
    for dev in devs:
        np.testing.assert_array_equal(dev.assemble(k, copy_out=True), ref)
    assert free - torch.cuda.mem_get_info()[0] < 32 << 20  # a chunk set per context would take 8 MB each
    for precision in ("fp64", "mixed"):
        ref = devs[0].assemble(k, precision=precision, copy_out=True)
        with ThreadPoolExecutor(len(devs)) as pool:
            for Z in pool.map(lambda d: d.assemble(k, precision=precision, copy_out=True), devs):
                np.testing.assert_array_equal(Z, ref)
    for dev in devs:
        dev.close()
    # kept for a context that follows; given back by one that did not use
    # them, and made again
    for calls in (1, 0, 4):
        dev = EFIEDevice(mesh, rwg)
        for _ in range(calls):
            np.testing.assert_array_equal(dev.assemble(k, precision="mixed", copy_out=True), ref)
        dev.close()
