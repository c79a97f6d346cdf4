"""A mesh whose arrays are too large for the memory pools: copies of a small one,
each smoothed to the small one's normals and with its sharp edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_copies_of_a_small_mesh(gpu_lib):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.geom import Radians
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.meshops import DeviceMesh
    from fauxgl_gb300.shapes import sphere_positions

    copies = 200  # 4.1 M triangles: 590 MB of positions and normals on the device
    pos = np.round(scenes.displace(sphere_positions(5), 3) * 2.0 ** 20) / 2.0 ** 20  # shifts stay exact
    nrm = np.cross(pos[:, 1] - pos[:, 0], pos[:, 2] - pos[:, 0])
    nrm = np.repeat((nrm / np.linalg.norm(nrm, axis=1, keepdims=True))[:, None, :], 3, 1)
    shift = np.zeros((copies, 1, 1, 3))
    shift[:, 0, 0, 0] = 4.0 * np.arange(copies)

    def run(m):
        d = DeviceMesh.upload(m)
        d.SmoothNormalsThreshold(Radians(40.0))
        return d.download().tri_nrm, d.SharpEdges(Radians(30.0)).download().line_pos

    small, edges = run(Mesh(pos, nrm))
    n, e = run(Mesh((pos[None] + shift).reshape(-1, 3, 3), np.tile(nrm, (copies, 1, 1))))
    assert len(edges) > 100
    assert np.array_equal(n.reshape(copies, -1, 3, 3).view(np.uint64),
                          np.broadcast_to(small, (copies,) + small.shape).copy().view(np.uint64))
    assert np.array_equal(e.reshape(copies, -1, 2, 3), edges[None] + shift)
