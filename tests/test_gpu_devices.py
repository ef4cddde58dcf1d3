"""Contexts on several devices of one process: kernels with raised shared-memory
limits launch on each of them."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _device_count():
    try:
        import torch
        return torch.cuda.device_count()
    except Exception:
        return 0


@pytest.mark.skipif(_device_count() < 2, reason="needs two GPUs")
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_each_device_gives_the_same(precision):
    from diffmom_b200 import EFIEDevice, build_rwg, make_rect_plate
    mesh = make_rect_plate(0.1, 0.1, 20, 20)
    rwg = build_rwg(mesh)
    rng = np.random.default_rng(0)
    B = np.asfortranarray(rng.standard_normal((rwg.nedges, 64)) + 1j * rng.standard_normal((rwg.nedges, 64)))
    out = []
    for device in range(2):
        dev = EFIEDevice(mesh, rwg, device=device)
        Z = dev.assemble(2 * math.pi / 0.1, precision=precision, copy_out=True)
        dev.build_nearfield(math.inf, "lu")
        out.append([Z, dev.nf_apply(B[:, 0]), dev.nf_apply(B[:, :16]), dev.nf_apply(B), dev.matvec(B)])
        dev.build_local(0.02)
        out[-1].append(dev.nf_apply(B[:, 0]))
        dev.close()
    for first, second in zip(*out):
        np.testing.assert_array_equal(second, first)
