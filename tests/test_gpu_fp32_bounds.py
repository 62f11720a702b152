"""The FP32 point-triangle distance behind the running upper bounds and the
within-tolerance verdicts: with the evaluation band its callers add (128 u span
+ 1e-8) it is never below the FP64 distance of the same points, wherever they
lie.  Triangles of 1e-5 .. 1e-2 m, half of them slivers, 1e-2 .. 10 m from the
origin, points a few sizes away; the FP32 coordinates are taken as exact, so no
placement bound hides the evaluation's own error."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KU = 2.0 ** -24
SOURCE = """
#include "kgpu_dist32.cuh"
using namespace kgpu;
__global__ void k(const float* x, int n, float* out)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float3 v[4];
  for (int k = 0; k < 4; ++k) v[k] = make_float3(x[12 * i + 3 * k], x[12 * i + 3 * k + 1], x[12 * i + 3 * k + 2]);
  out[i] = sqrtf(pt_tri2_32(v[0], v[1], v[2], v[3]));
}
extern "C" int run(const float* x, int n, float* out)
{
  k<<<(n + 255) / 256, 256>>>(x, n, out);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    import torch
    from klampt_gb300 import build
    d = tmp_path_factory.mktemp("fp32")
    src, lib = str(d / "probe.cu"), str(d / "probe.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", build.CSRC,
                    "-I", os.path.join(build.ROOT, "include"), src, "-o", lib], check=True, capture_output=True)
    fn = ctypes.CDLL(lib).run

    def call(x):
        xd = torch.as_tensor(x).cuda()
        out = torch.empty(len(x), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        assert fn(ctypes.c_void_p(xd.data_ptr()), len(x), ctypes.c_void_p(out.data_ptr())) == 0
        return out.cpu().numpy().astype(np.float64)
    return call


def _point_triangle(p, T):
    """Distance of points p [n, 3] to triangles T [n, 3, 3], in FP64: the plane
    where the foot is inside, otherwise the nearest edge."""
    n = np.cross(T[:, 1] - T[:, 0], T[:, 2] - T[:, 0])
    h = ((p - T[:, 0]) * n).sum(1) / (n * n).sum(1)
    foot = p - h[:, None] * n
    inside = np.ones(len(p), bool)
    best = np.full(len(p), np.inf)
    for k in range(3):
        a, e = T[:, k], T[:, (k + 1) % 3] - T[:, k]
        inside &= (np.cross(e, foot - a) * n).sum(1) >= 0
        t = np.clip(((p - a) * e).sum(1) / (e * e).sum(1), 0, 1)
        best = np.minimum(best, np.linalg.norm(p - a - t[:, None] * e, axis=1))
    return np.where(inside, np.minimum(best, np.linalg.norm(p - foot, axis=1)), best)


@pytest.mark.parametrize("size", [1e-5, 1e-4, 1e-2])
@pytest.mark.parametrize("far", [1e-2, 0.3, 10.0])
def test_fp32_point_triangle_distance_is_an_upper_bound(run, size, far):
    rng = np.random.default_rng(int(far * 100))
    n = 1 << 20
    c = rng.normal(size=(n, 1, 3))
    c = c / np.linalg.norm(c, axis=-1, keepdims=True) * far
    x = np.concatenate([c + rng.uniform(-3, 3, (n, 1, 3)) * size, c + rng.uniform(-1, 1, (n, 3, 3)) * size], 1)
    x[::2, 3] = x[::2, 2] + (x[::2, 3] - x[::2, 2]) * np.exp(rng.uniform(np.log(1e-4), 0, (len(x[::2]), 1)))
    x = x.astype(np.float32)
    x64 = x.astype(np.float64)
    area = np.linalg.norm(np.cross(x64[:, 2] - x64[:, 1], x64[:, 3] - x64[:, 1]), axis=1)
    keep = area > 1e-5 * size * size  # (the FP64 reference divides by it)
    x, x64 = np.ascontiguousarray(x[keep]), x64[keep]
    out = run(x.reshape(-1, 12))
    span = (x64.max(1) - x64.min(1)).max(1)
    # (1e-14 of the coordinates: the FP64 reference's own rounding)
    assert (out + 128 * KU * span + 1e-8 >= _point_triangle(x64[:, 0], x64[:, 1:]) - 1e-14 * far).all()
