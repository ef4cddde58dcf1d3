"""The bounded-wait error path, exercised without any GPU fault: the triangular
sweeps of a near-field factor wait for values published by earlier CTAs, and the
tiles of a factorisation panel for its diagonal tiles; with DMB_OPT_SPIN_LIMIT = 0
a waiting CTA gives up at its first poll, records the error bit and returns.  The call must fail with
DMB_ERR_TIMEOUT (DeviceWaitTimeout), and the next call on the same context,
with the default limit, must give the right answer."""
import math

import numpy as np
import pytest

import oracle as orc
from diffmom_b200 import DeviceWaitTimeout, EFIEDevice, build_rwg, make_rect_plate, rwg_centers

pytestmark = pytest.mark.gpu


def test_chain_wait_expires_and_context_recovers():
    m = make_rect_plate(0.1, 0.1, 24, 24)   # 1,680 RWG: seven 256-row blocks of a sweep
    r = build_rwg(m)
    k = 2 * math.pi / 0.1
    dev = EFIEDevice(m, r)
    dev.assemble(k, precision="fp64")
    cutoff = 0.3 * 0.1
    dev.build_nearfield(cutoff, "lu")
    x = np.random.default_rng(3).standard_normal(r.nedges) * (1 + 0.25j)
    dev.set_option("spin_limit", 0)
    with pytest.raises(DeviceWaitTimeout):
        dev.nf_apply(x)
    dev.set_option("spin_limit", -1)
    y = dev.nf_apply(x)
    c = orc.OracleCache(m, r, 3)
    Znf = orc.nearfield_matrix(c.assemble_z(k), rwg_centers(m, r), cutoff)
    ref = np.linalg.solve(Znf, x)
    err = np.linalg.norm(y - ref) / np.linalg.norm(ref)
    print(f"after the expired wait: near-field apply vs oracle {err:.2e}")
    assert err < 1e-10
    # and a solve on the same context still converges
    v = c.plane_wave_rhs([0, 0, -k], 1.0, [1, 0, 0])
    I, st = dev.gmres(v, tol=1e-8, maxiter=200, preconditioner=dev.preconditioner)
    assert st.solved and st.true_residual <= 1e-8
    dev.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_no_expired_wait_is_lost(precision):
    """Limits at which some of a solve's sweeps expire and others do not: the
    solve fails, or gives what it gives without a limit."""
    m = make_rect_plate(0.1, 0.1, 18, 20)
    dev = EFIEDevice(m, build_rwg(m))
    dev.assemble(2 * math.pi / 0.1, precision=precision)
    P = dev.build_nearfield(0.03, "lu")
    dev.set_option("true_residual", 0)
    b = np.random.default_rng(3).standard_normal(dev.N) + 0j

    def solve():
        return dev.gmres(b, tol=1e-6, maxiter=60, preconditioner=P, check_gmres_convergence=False)[0]

    ref, expired = solve(), 0
    for limit in [int(1.25 ** e) for e in range(8, 44)]:  # 5 to 14,000 polls
        for _ in range(3):
            dev.set_option("spin_limit", limit)
            try:
                np.testing.assert_array_equal(solve(), ref)
            except DeviceWaitTimeout:
                expired += 1
    dev.set_option("spin_limit", -1)
    np.testing.assert_array_equal(solve(), ref)
    dev.close()
    assert expired > 0


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_factorisation_wait_expires_and_context_recovers(precision):
    """The tiles of a 256-wide panel wait for its diagonal tiles."""
    m = make_rect_plate(0.1, 0.1, 20, 23)   # 1,337 RWG: six panels, two block columns
    dev = EFIEDevice(m, build_rwg(m))
    Z = dev.assemble(2 * math.pi / 0.1, precision=precision, copy_out=True)
    dev.set_option("spin_limit", 0)
    with pytest.raises(DeviceWaitTimeout):
        dev.build_nearfield(math.inf, "lu")
    dev.set_option("spin_limit", -1)
    dev.build_nearfield(math.inf, "lu")
    b = np.random.default_rng(3).standard_normal(dev.N) + 0j
    x = dev.nf_apply(b)
    dev.close()
    # N-term sums of the factor's precision, twice (factor and sweeps)
    eps = 2.0 ** -52 if precision == "fp64" else 2.0 ** -23
    assert np.linalg.norm(Z @ x - b) < Z.shape[0] * eps * np.linalg.norm(Z) * np.linalg.norm(x)
