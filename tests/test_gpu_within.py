"""Geometry pairs within a tolerance: FP32 settles most triangle pairs, the
others are decided in FP64 on the features that may matter.  Tolerances at and
one step beside a query's own distance, far below and far above the triangles'
size, with margins, and triangles without area or much longer than wide.
Verdicts equal the FP64 oracle's."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 4


@pytest.fixture(scope="module")
def built():
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()


def _soup(n, rng, shape):
    V = rng.uniform(-0.05, 0.05, (n, 1, 3)) + rng.uniform(-0.04, 0.04, (n, 3, 3))
    if shape == "sliver":
        V[:, 2] = V[:, 1] + rng.uniform(-1e-6, 1e-6, (n, 3))
    elif shape == "flat":
        V[::2, 2] = 0.25 * V[::2, 0] + 0.75 * V[::2, 1]
        V[1::4, 1] = V[1::4, 0]
    elif shape == "tiny":
        V = V[:, :1] + rng.uniform(-1e-5, 1e-5, (n, 3, 3))
    return V.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3)


def _placements(rng, n, spread):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                  2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                  2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1)
    return np.ascontiguousarray(np.concatenate([R, rng.uniform(-spread, spread, (n, 3))], 1))


@pytest.mark.parametrize("margins", [(0.0, 0.0), (0.003, 0.01)])
@pytest.mark.parametrize("shape", ["plain", "sliver", "flat", "tiny"])
@pytest.mark.parametrize("n", [1, 9, 60])
def test_within(built, n, shape, margins):
    from klampt_gb300.engine import Geometry
    from oracle.oracle_py import GeomPairOracle
    rng = np.random.default_rng(n)
    A, B = _soup(n, rng, shape), _soup(n + 3, rng, "plain")
    Ta, Tb = _placements(rng, 300, 0.15), _placements(rng, 300, 0.15)
    ga, gb = Geometry(*A), Geometry(*B)
    ga.set_margin(margins[0])
    gb.set_margin(margins[1])
    o = GeomPairOracle(A, B, margin_a=margins[0], margin_b=margins[1])
    d, _, _, _ = o.distance(Ta, Tb, nthreads=NT)
    own = d[d > 0][:4]
    tols = [0.0, 1e-9, 1e-4, 0.02, 0.2, 10.0] + [f(x) for x in own for f in
                                                 (float, lambda x: np.nextafter(x, 0), lambda x: np.nextafter(x, 1))]
    for tol in tols:
        ho = o.collide(Ta, Tb, tol=float(tol), nthreads=NT)
        assert np.array_equal(ga.collide(gb, Ta, Tb, tol=float(tol)).cpu().numpy(), ho), tol
    ga.close()
    gb.close()
