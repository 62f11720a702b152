"""Limits of a soft-min call: more waypoints than its launches can count are
refused before anything is launched."""

import ctypes

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    from klampt_gb300 import build
    build.build()
    from klampt_gb300.engine import World
    robot = sc.arm(2, rings=1, segments=4)
    w = World(sc.env_from_objects("one", [sc.box_mesh((0.5, 0, 0.3), (0.05,) * 3)]), [robot])
    yield w
    w.close()


@pytest.mark.parametrize("T, Wn", [(65536, 65536), (2 ** 31 - 1, 2), (46341, 46341), (2 ** 31 - 1, 2 ** 31 - 1),
                                   (1, 2 ** 31 - 1), (2 ** 31 - 8192, 1)])
def test_more_waypoints_than_fit_are_refused(world, T, Wn):
    import torch
    from klampt_gb300 import _kgpu
    x = torch.zeros(64, dtype=torch.float64, device="cuda")  # never touched by a refused call
    p = ctypes.c_void_p(x.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    st = _kgpu.load().kgpu_softmin_grad(world.handle, 0, p, T, Wn, ctypes.c_double(0.01), p, p, stream)
    assert st == _kgpu.KGPU_ERR_INVALID and "waypoints" in _kgpu.last_error()
    q = np.zeros((3, 5, 2), np.float32)  # the world answers on
    assert np.isfinite(world.softmin(q, 0.01)[0].cpu().numpy()).all()
