"""Limits of a soft-min call: more waypoints than its launches can count are
refused before anything is launched; with little device memory left the call
takes smaller chunks, with the same results to the bit."""

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


def test_little_device_memory():
    import torch
    from klampt_gb300 import build
    build.build()
    from klampt_gb300.engine import World
    rng = np.random.default_rng(3)
    robot = sc.arm(2, rings=1, segments=4)
    env = sc.env_from_objects("boxes", sc.random_boxes(150, rng, -0.8, 0.8, 0.01, 0.03))
    q = torch.as_tensor(rng.uniform(robot.qmin, robot.qmax, (260, 33, 2)).astype(np.float32)).cuda()
    roomy, w = World(env, [robot]), World(env, [robot])
    ref = roomy.softmin(q, 0.02)
    roomy.close()
    w.softmin(q[:1, :1], 0.02)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    for left in (80 << 20, 24 << 20):  # 8,580 waypoints ask for 126 MB
        hog = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
        try:
            L, G = w.softmin(q, 0.02)
            assert torch.equal(L, ref[0]) and torch.equal(G, ref[1])
        finally:
            del hog
            torch.cuda.empty_cache()
    w.close()
