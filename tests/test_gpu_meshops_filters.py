"""Smoothing and sharp edges where the FP32 and cosine filters must leave the
decision to FP64: dot products at the threshold, normals of extreme lengths,
large groups, angles at and beyond the ends of acos's range. Bit for bit
against the oracle."""
import math

import numpy as np
import pytest

from fauxgl_gb300 import scenes
from fauxgl_gb300.mesh import Mesh
from fauxgl_gb300.shapes import NewCone, NewCube, cylinder_segments, sphere_positions
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.uint64)


def fan(n, normals):
    """n triangles around one point, corner normals given per triangle."""
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(a), np.sin(a), 0 * a], -1)
    pos = np.stack([np.zeros((n, 3)), ring, np.roll(ring, -1, 0)], 1)
    return Mesh(pos, np.repeat(np.asarray(normals, dtype=np.float64)[:, None, :], 3, 1))


def normal_sets():
    rng = np.random.RandomState(3)
    unit = rng.normal(size=(40, 3))
    unit /= np.linalg.norm(unit, axis=1, keepdims=True)
    tilt = np.array([[math.sin(t), 0.0, math.cos(t)] for t in np.radians([0, 30, 30 + 1e-7, 30 - 1e-7, 60, 15])])
    return {
        "axes": np.array([[1, 0, 0], [0, 1, 0], [0, 0, 1], [-1, 0, 0], [1, 0, 0], [0, 0, -1]], dtype=float),
        "tilted": tilt,
        "long": unit * 10.0 ** rng.uniform(-25, 25, (40, 1)),
        "zeros": np.concatenate([np.zeros((3, 3)), unit[:4]]),
        "odd": np.array([[np.nan, 0, 0], [np.inf, 0, 0], [0, 0, 1], [0, 0, 1], [1e300, 0, 0]]),
        "sixteen": unit[:16] * 0.05 + [0, 0, 1],
        "seventeen": unit[:17] * 0.05 + [0, 0, 1],
    }


@pytest.mark.parametrize("name", sorted(normal_sets()))
@pytest.mark.parametrize("degrees", [0.0, 30.0, 60.0, 90.0, 180.0])
def test_smoothing(gpu_lib, name, degrees):
    from fauxgl_gb300.meshops import DeviceMesh

    m = fan(len(normal_sets()[name]), normal_sets()[name])
    thr = math.radians(degrees)
    d = DeviceMesh.upload(m)
    d.SmoothNormalsThreshold(thr)
    want = O.smooth_normals_threshold(m.tri_pos, m.tri_nrm, math.cos(thr))
    got = d.download().tri_nrm
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got).ravel(), nan.ravel())
    assert np.array_equal(bits(got).ravel()[~nan.ravel()], bits(want).ravel()[~nan.ravel()])


@pytest.mark.parametrize("angle", [-1.0, 0.0, 1e-9, 0.5, 3.0, math.pi, 4.0, float("nan")])
def test_sharp_edges(gpu_lib, angle):
    from fauxgl_gb300.meshops import DeviceMesh

    folded = np.array([[[0, 0, 0], [1, 0, 0], [0, 1, 0]], [[1, 0, 0], [0, 0, 0], [0, 1, 0]]], dtype=float)
    for pos in (NewCube().tri_pos, NewCone(15, True).tri_pos, cylinder_segments(64).tri_pos, folded,
                scenes.displace(sphere_positions(3), 4)):
        got = DeviceMesh.upload(Mesh(pos)).SharpEdges(angle).download()
        want = O.sharp_edges(pos, angle)
        assert got.nline == want.shape[0]
        assert np.array_equal(bits(got.line_pos).ravel(), bits(want).ravel())
