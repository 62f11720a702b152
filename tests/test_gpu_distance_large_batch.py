"""A distance batch whose result indices pass 2^31 (six numbers per
configuration, 358 M configurations of a one-link arm): the last results are
those of a small batch."""

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu


def test_results_beyond_2_31_entries():
    import torch
    from klampt_gb300 import build
    build.build()
    from klampt_gb300.engine import World
    B = 2 ** 31 // 6 + 100
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    robot = sc.arm(1, rings=1, segments=4)
    w = World(sc.env_from_objects("one", [sc.box_mesh((0.3, 0, 0.3), (0.05,) * 3)]), [robot])
    tail = torch.as_tensor(np.random.default_rng(0).uniform(robot.qmin, robot.qmax, (200, 1)).astype(np.float32)).cuda()
    cutoff = float(w.distance(tail, 10.0)[0].median())  # half of them find nothing
    ref = [x.cpu().numpy() for x in w.distance(tail, cutoff, want_grad=False)[:3]]
    none = np.flatnonzero(ref[1][:, 0] < 0)
    assert 0 < len(none) < 200
    q = torch.zeros((B, 1), dtype=torch.float32, device="cuda")
    q[:] = tail[int(none[0])]
    q[-200:] = tail
    out = w.distance(q, cutoff, want_grad=False)[:3]
    assert all(np.array_equal(x[-200:].cpu().numpy(), r) for x, r in zip(out, ref))
    assert all(bool((x == x[0]).all()) for x in (out[0][:-200], out[1][:-200, 0], out[2][:-200, 0]))
    w.close()
    del q, out
    torch.cuda.empty_cache()
