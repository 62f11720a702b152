"""The FP64 finalisation of distances evaluates only the triangle features
that FP32 cannot rule out: values, closest points and elements stay those of
the whole canonical function (the FP64 oracle), where FP32 feature distances
are least exact — nearly parallel edges, slivers, triangles far smaller than
their distance, near contact.  The two sides do the same FP64 operations, so
equality is exact."""

import os

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 4


def _rotation(axis, angle):
    axis = axis / np.linalg.norm(axis)
    K = np.array([[0, -axis[2], axis[1]], [axis[2], 0, -axis[0]], [-axis[1], axis[0], 0]])
    return np.eye(3) + np.sin(angle) * K + (1 - np.cos(angle)) * K @ K


def _placements(rng, n, tilt, offset):
    """Transforms rotated by a log-uniform angle in `tilt`, moved by up to a
    log-uniform distance in `offset` along a random axis on top of x."""
    T = np.zeros((n, 12))
    for k in range(n):
        a = np.exp(rng.uniform(*np.log(tilt)))
        T[k, :9] = _rotation(rng.normal(size=3), a).ravel()
        T[k, 9:] = rng.normal(size=3) * 0.02
        T[k, 9] += np.exp(rng.uniform(*np.log(offset)))
    return T


CASES = {
    # two boxes a hair apart, edges parallel to within 1e-7 .. 1e-2 rad
    "parallel_boxes": (lambda: sc.box_mesh((0, 0, 0), (0.1, 0.1, 0.1)), lambda: sc.box_mesh((0.2, 0, 0), (0.1, 0.1, 0.1)),
                       (1e-7, 1e-2), (1e-6, 1e-1)),
    # long slivers against an icosphere and against each other
    "sliver_sphere": (lambda: sc.cylinder_mesh(0.05, 1.5, 64, 1), lambda: sc.icosphere_mesh((0.2, 0, 0.5), 0.1, 2),
                      (1e-3, 3.0), (1e-4, 0.3)),
    "sliver_sliver": (lambda: sc.cylinder_mesh(0.03, 1.0, 48, 1), lambda: sc.cylinder_mesh(0.03, 1.0, 48, 1),
                      (1e-6, 3.0), (0.06, 0.4)),
    # triangles of 0.1 mm a metre away
    "tiny_far": (lambda: sc.icosphere_mesh((0, 0, 0), 1e-3, 2), lambda: sc.cylinder_mesh(0.05, 0.3, 32, 16),
                 (1e-3, 3.0), (0.2, 2.0)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_finalised_features_match_oracle(name):
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()
    from klampt_gb300.engine import Geometry
    ma, mb, tilt, offset = CASES[name]
    A, B = ma(), mb()
    rng = np.random.default_rng(len(name))
    n = 512
    Ta = np.tile(np.array([1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0.0]), (n, 1))
    Tb = _placements(rng, n, tilt, offset)
    d_o, cp_o, el_o, _ = oracle_py.GeomPairOracle(A, B).distance(Ta, Tb, nthreads=NT)[:4]
    d, cp, el, _ = (x.cpu().numpy() for x in Geometry(*A).distance(Geometry(*B), Ta, Tb))
    assert np.array_equal(d, d_o)
    assert np.array_equal(el, el_o)
    assert np.array_equal(cp, cp_o)
    assert (d_o > 0).any()
