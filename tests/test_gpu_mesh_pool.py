"""Meshes and their temporaries from the device memory pool: calls from several
threads at once, and meshes that outlive the calls that made them, give the
results of one call after the other."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh_results(detail, seed):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.geom import Radians
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.meshops import DeviceMesh
    from fauxgl_gb300.shapes import sphere_positions

    pos = scenes.displace(sphere_positions(detail), seed)
    d = DeviceMesh.upload(Mesh(pos, pos))
    lines = d.SharpEdges(Radians(20.0))
    outline = d.Silhouette((2.0, 1.0, 0.5), 1e-3)
    d.SmoothNormalsThreshold(Radians(40.0))
    m, l, o = d.download(), lines.download(), outline.download()
    return [m.tri_pos, m.tri_nrm, l.line_pos, o.line_pos]


@pytest.mark.parametrize("threads", [2, 12])  # fewer and more than the kept streams
def test_threads_give_the_results_of_one(gpu_lib, threads):
    jobs = [(2 + i % 4, i) for i in range(3 * threads)]
    want = [_mesh_results(*j) for j in jobs]
    got, errors = [None] * len(jobs), []

    def work(t):
        try:
            for i in range(t, len(jobs), threads):
                got[i] = _mesh_results(*jobs[i])
        except Exception as e:  # reported by the assertion below
            errors.append(e)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
    for a, b in zip(want, got):
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=True)
