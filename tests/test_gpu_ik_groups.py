"""Several IK problems share a warp: each must come out exactly as it does
alone.  Robots of every group width (8, 16, 32 lanes), position with and
without rotation, one link for all or one per problem, and batches around the
edges of a warp and of a block's share, problems that reach the iteration
limit among them."""

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def worlds():
    from klampt_gb300 import build
    build.build()
    from klampt_gb300.engine import World
    env = sc.env_from_objects("far", [sc.box_mesh((9, 9, 9), (0.1, 0.1, 0.1))])
    robots = [sc.arm(7, rings=1), sc.dual_arm(rings=1), sc.humanoid()]
    w = World(env, robots)
    yield robots, w
    w.close()


@pytest.mark.parametrize("robot", [0, 1, 2])
@pytest.mark.parametrize("rotation", [False, True])
@pytest.mark.parametrize("B", [1, 3, 33, 1300])
def test_batch_equals_single_solves(worlds, robot, rotation, B):
    robots, w = worlds
    r = robots[robot]
    L = r.num_links
    rng = np.random.default_rng(B + robot)
    link = rng.integers(max(0, L - 4), L, B).astype(np.int32) if B > 1 else L - 1
    links = np.broadcast_to(link, (B,))
    qt = rng.uniform(np.maximum(r.qmin, -2.5), np.minimum(r.qmax, 2.5), (B, L)).astype(np.float32)
    T = w.fk(qt, robot=robot).cpu().numpy()[np.arange(B), links]
    pl = np.float32([0, 0, 0.1])
    pt = (np.einsum("bij,j->bi", T[:, :9].reshape(B, 3, 3), pl) + T[:, 9:]).astype(np.float32)
    pt[::17] += 5.0  # out of reach
    q0 = (qt + rng.normal(0, 0.4, qt.shape)).astype(np.float32)
    Rt = T[:, :9].copy() if rotation else None
    kw = dict(max_iters=60, tol=1e-4, robot=robot)
    q, ok, res, it = (x.cpu().numpy() for x in w.ik_solve(q0, link, pl[None], pt, Rtarget=Rt, **kw))
    assert ok.mean() > 0.5 or B == 1
    for b in range(0, B, max(1, B // 60)):
        q1, ok1, res1, it1 = (x.cpu().numpy() for x in w.ik_solve(
            q0[b:b + 1], int(links[b]), pl[None], pt[b:b + 1], Rtarget=None if Rt is None else Rt[b:b + 1], **kw))
        assert np.array_equal(q[b], q1[0]) and ok[b] == ok1[0] and res[b] == res1[0] and it[b] == it1[0], b
