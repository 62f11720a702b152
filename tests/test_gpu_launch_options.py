"""Launch options that the caller sets hold for small batches too."""

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    from klampt_gb300 import build
    build.build()
    from klampt_gb300.engine import World
    robot = sc.arm(7, rings=32)
    w = World(sc.sphere_field(np.random.default_rng(1001), n=2000), [robot])
    yield robot, w
    w.close()


def test_job_flush_holds_for_single_configurations(world):
    """The triangle pairs that one configuration's warp tests depend on how
    many jobs it collects (one warp per configuration, so the count is the
    same from run to run)."""
    robot, w = world
    q = sc.uniform_configs(robot, 100, np.random.default_rng(0))

    def tested(flush):
        w.set_option("job_flush", flush)
        assert w.get_option("job_flush") == flush
        out = []
        for k in range(len(q)):
            w.reset_stats()
            w.is_feasible(q[k:k + 1])
            out.append(w.stats()["tri_pairs"])
        return out

    counts = {f: tested(f) for f in (32, 64)}
    assert counts[64] == tested(64)
    assert counts[32] != counts[64]


def _kernel_grids(plan):
    """Blocks of the 256-thread kernels in a plan's graph (the plan starts with
    the pointers to its world and its graph)."""
    import ctypes
    cu = ctypes.CDLL("libcuda.so.1")
    graph = ctypes.c_void_p(ctypes.cast(plan.handle, ctypes.POINTER(ctypes.c_void_p))[1])
    n = ctypes.c_size_t(0)
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    grids = []
    for node in nodes:
        kind = ctypes.c_int(-1)
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 0:  # a kernel: function pointer, grid, block, ...
            p = (ctypes.c_uint32 * 64)()
            assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), p) == 0
            if p[5] == 256:
                grids.append(p[2])
    return grids


def test_blocks_per_sm_holds_for_few_edges(world):
    import torch
    from klampt_gb300.engine import World
    robot, w = world
    qa, qb, n = (torch.as_tensor(np.ascontiguousarray(x)).cuda()
                 for x in sc.random_edges(robot, 24, np.random.default_rng(1), max_steps=100))
    out = torch.empty(24, dtype=torch.int32, device="cuda")
    sms = int(w.get_option("num_sms"))
    ref = w.check_edges(qa, qb, n)
    fresh = World(sc.env_from_objects("one", [sc.box_mesh((0.5, 0, 0.3), (0.05,) * 3)]), [robot])
    plan = fresh.edge_plan(qa, qb, n, out)
    assert 2 * sms in _kernel_grids(plan) and 3 * sms not in _kernel_grids(plan)  # not set: 2 for so few
    plan.close()
    fresh.close()
    for k in (4, 3, 2):
        w.set_option("blocks_per_sm", k)
        plan = w.edge_plan(qa, qb, n, out)
        assert k * sms in _kernel_grids(plan)
        plan.launch()
        w.sync()
        assert torch.equal(out, ref)
        plan.close()
