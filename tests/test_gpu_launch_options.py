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
