"""Distances of meshes whose triangles have no area: the canonical function
reports a contact of some such pairs that are apart (its overlap axes vanish),
and every distance query that reaches one reports it as the FP64 oracle does —
single points, collinear and duplicate vertices, and segments in one plane."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(kind, n, rng):
    V = rng.uniform(-0.1, 0.1, (n, 3, 3))
    if kind == "points":
        V[:] = V[:, :1]
    elif kind == "line":
        V[:, 2] = 0.25 * V[:, 0] + 0.75 * V[:, 1]
    else:
        V[:, 2] = V[:, 1]
    if kind == "coplanar":
        V[:, :, 2] = 0.0
    return V.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3)


@pytest.mark.parametrize("kind", ["points", "line", "duplicate", "coplanar"])
@pytest.mark.parametrize("n", [1, 4, 30])
def test_flat_triangles_match_oracle(kind, n):
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()
    from klampt_gb300.engine import Geometry
    rng = np.random.default_rng(n)
    A, B = _soup(kind, n, rng), _soup(kind, n + 2, rng)
    a, t = rng.uniform(0, 2 * np.pi, 200), rng.uniform(-0.3, 0.3, (200, 3))
    o, z = np.ones(200), np.zeros(200)
    Tb = np.stack([np.cos(a), -np.sin(a), z, np.sin(a), np.cos(a), z, z, z, o, *t.T], 1)
    if kind == "coplanar":
        Tb[:, 11] = 0.0
    Ta = np.array([[1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0.0]])
    d_o = oracle_py.GeomPairOracle(A, B).distance(np.repeat(Ta, 200, 0), Tb, nthreads=os.cpu_count() or 4)[0]
    d = Geometry(*A).distance(Geometry(*B), Ta, Tb)[0].cpu().numpy()
    assert np.array_equal(d, d_o)
    assert (d_o == 0).all() == (kind in ("points", "coplanar"))
