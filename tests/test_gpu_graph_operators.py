"""Captured GMRES iterations on a device whose operator, factor or options
change between solves: every solve must give bitwise what direct launches
give.  Repeated often enough that each state meets its iterations eagerly,
captured and replayed while the buffers no longer grow."""
import math

import numpy as np
import pytest

from diffmom_b200 import _native as nat
from diffmom_b200 import DeviceWaitTimeout, EFIEDevice, build_aca_operator, build_rwg, make_rect_plate

pytestmark = pytest.mark.gpu

K = 2 * math.pi / 0.1
ROUNDS = 4


def _plate(nx, ny):
    mesh = make_rect_plate(0.005 * nx, 0.005 * ny, nx, ny)
    return mesh, build_rwg(mesh)


def _rhs(n, columns=None):
    rng = np.random.default_rng(5)
    shape = (n,) if columns is None else (n, columns)
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


def _alternating(states, nx=14, ny=15):
    """ROUNDS times the solves `states(device, mesh, rwg)` yields, with graphs
    and without."""
    runs = []
    for graphs in (0, 1):
        mesh, rwg = _plate(nx, ny)
        dev = EFIEDevice(mesh, rwg)
        dev.set_option("gmres_graphs", graphs)
        runs.append([x.copy() for _ in range(ROUNDS) for x in states(dev, mesh, rwg)])
        dev.close()
    assert len(runs[0]) == len(runs[1])
    for direct, replayed in zip(*runs):
        np.testing.assert_array_equal(replayed, direct)


def test_hmatrix_forward_and_adjoint():
    def states(dev, mesh, rwg):
        if not hasattr(dev, "op"):
            dev.op = build_aca_operator(mesh, rwg, K, leaf_size=16, aca_tol=1e-4, device=dev)
            dev.pc = dev.op.build_nearfield("lu")
        for adjoint in (False, True):
            yield dev.op.gmres(_rhs(dev.N), tol=1e-9, maxiter=60, preconditioner=dev.pc, adjoint=adjoint,
                               check_gmres_convergence=False)[0]
    _alternating(states)


def test_dense_and_hmatrix_at_two_frequencies():
    def states(dev, mesh, rwg):
        if not hasattr(dev, "op"):
            dev.op = build_aca_operator(mesh, rwg, K, leaf_size=16, device=dev)
            dev.assemble(1.1 * K)
        for operator in (0, 1):
            dev.ctx.call("dmb_set_option", nat.OPT_OPERATOR, operator)
            yield dev.gmres(_rhs(dev.N), tol=1e-8, maxiter=40, check_gmres_convergence=False)[0]
    _alternating(states)


@pytest.mark.parametrize("columns", [None, 3])
def test_factor_precisions(columns):
    def states(dev, mesh, rwg):
        if not hasattr(dev, "op"):
            dev.op = build_aca_operator(mesh, rwg, K, leaf_size=16, device=dev)
        for precision in ("fp64", "mixed"):
            P = dev.op.build_nearfield("lu", precision)
            yield dev.op.gmres(_rhs(dev.N, columns), tol=1e-8, maxiter=60, preconditioner=P)[0]
    _alternating(states)


def test_hmatrix_plans():
    """Two plans of one mesh on the same device: another number of blocks,
    low-rank blocks and leaves."""
    def states(dev, mesh, rwg):
        for leaf_size, eta in ((8, 1.5), (40, 1.0)):
            op = build_aca_operator(mesh, rwg, K, leaf_size=leaf_size, eta=eta, device=dev)
            P = op.build_nearfield("diag")
            yield op.gmres(_rhs(dev.N), tol=1e-8, maxiter=40, preconditioner=P, check_gmres_convergence=False)[0]
    _alternating(states)


@pytest.mark.parametrize("side", ["left", "right"])
def test_packed_operands_follow_the_matrix(side):
    """Tensor-core products and sweeps of a batch small enough to be captured
    use operands packed once per matrix and once per factor."""
    def states(dev, mesh, rwg):
        dev.set_option("tc_min_rhs", 16)
        for k in (K, 1.2 * K):
            dev.assemble(k, precision="mixed")
            P = dev.build_nearfield(math.inf, "lu")
            for _ in range(3):  # captured while the packed operands are up to date
                x, st = dev.gmres(_rhs(dev.N, 16), tol=1e-6, maxiter=30, preconditioner=P, precond_side=side)
                assert st.solved and st.niter < 10
                yield x
    _alternating(states)


def test_spin_limit_reaches_captured_sweeps():
    mesh, rwg = _plate(20, 23)
    dev = EFIEDevice(mesh, rwg)
    dev.assemble(K)
    P = dev.build_nearfield(math.inf, "lu")
    solve = lambda: dev.gmres(_rhs(dev.N), tol=1e-8, maxiter=20, preconditioner=P)[0]  # noqa: E731
    x = [solve() for _ in range(ROUNDS)]
    dev.set_option("spin_limit", 0)
    with pytest.raises(DeviceWaitTimeout):
        solve()
    dev.set_option("spin_limit", -1)
    np.testing.assert_array_equal(solve(), x[0])
    dev.close()
