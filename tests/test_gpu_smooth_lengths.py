"""SmoothNormalsThreshold of normals from FP32's subnormal range beside very long
ones: their products lie at the threshold of a right angle though one of the two
is nothing in FP32. Bit for bit against the oracle."""
import math

import numpy as np
import pytest

from fauxgl_gb300.mesh import Mesh
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _normals(kind):
    rng = np.random.RandomState(4)
    if kind == "axis":
        return np.array([[1e30, 0, 0], [1e-46, 0, 0], [0, 1e-46, 0], [0, 3e29, 0], [-1e30, 0, 0]])
    n = rng.normal(size=(14, 3))
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    exponents = np.where(np.arange(14) % 2, rng.uniform(-48, -43, 14), rng.uniform(27, 31, 14))
    return n * 10.0 ** exponents[:, None]


@pytest.mark.parametrize("kind", ["axis", "any"])
@pytest.mark.parametrize("degrees", [60.0, 90.0, 120.0])
def test_short_beside_long(gpu_lib, kind, degrees):
    from fauxgl_gb300.meshops import DeviceMesh

    normals = _normals(kind)
    n = len(normals)
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(a), np.sin(a), 0 * a], -1)
    pos = np.stack([np.zeros((n, 3)), ring, np.roll(ring, -1, 0)], 1)
    m = Mesh(pos, np.repeat(normals[:, None, :], 3, 1))
    thr = math.radians(degrees)
    d = DeviceMesh.upload(m)
    d.SmoothNormalsThreshold(thr)
    want = O.smooth_normals_threshold(m.tri_pos, m.tri_nrm, math.cos(thr))
    got = d.download().tri_nrm
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(got[ok].view(np.uint64), want[ok].view(np.uint64))
