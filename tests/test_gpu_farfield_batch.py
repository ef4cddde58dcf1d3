"""Far fields of one and of many columns at the edges of the kernel's groups
(four directions, four columns, chunks of points) against the oracle."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quad_order", [1, 3, 7])
@pytest.mark.parametrize("ndir,nrhs", [(1, 1), (3, 1), (181, 1), (5, 2), (7, 5), (2, 259)])
def test_farfield_groups(ndir, nrhs, quad_order):
    import oracle as orc
    from diffmom_b200 import EFIEDevice, build_rwg, make_icosphere
    mesh = make_icosphere(0.05, 2)
    rwg = build_rwg(mesh)
    dev = EFIEDevice(mesh, rwg)
    rng = np.random.default_rng(ndir + nrhs)
    d = rng.standard_normal((ndir, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    k = 2 * math.pi / 0.1
    I = rng.standard_normal((rwg.nedges, nrhs)) + 1j * rng.standard_normal((rwg.nedges, nrhs))
    E = dev.farfield(d, np.asfortranarray(I) if nrhs > 1 else I[:, 0], k=k, quad_order=quad_order)
    dev.close()
    G = orc.OracleCache(mesh, rwg, quad_order).radiation_vectors(d, k)
    ref = (G.reshape(3 * ndir, -1) @ I).reshape(ndir, 3, nrhs).transpose(1, 0, 2)
    # two orders of the same FP64 sum: at most the number of terms times 2^-53
    # of the magnitudes, which random currents keep near the result's norm
    assert np.linalg.norm(E.reshape(3, ndir, nrhs) - ref) < 1e-13 * np.linalg.norm(ref)
