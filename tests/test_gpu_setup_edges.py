"""Sizes at which the setup and binning kernels change their form, against the
oracle: clipped triangles up to 2,048 a pass get a warp each, more of them a
thread each; the row starts' scan shares a grid with the bin matrix's, in tiles
of 2,048 primitives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(pos, w, h, vertex_colors):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.geom import Identity
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader
    from oracle import oracle as O

    rng = np.random.RandomState(5)
    mesh = Mesh(pos, rng.normal(size=pos.shape))
    ctx = NewContext(w, h)
    ctx.Cull = CullNone
    ctx.Shader = NewPhongShader(Identity(), scenes.LIGHT, scenes.EYE)
    if vertex_colors:
        mesh.tri_col = rng.uniform(0, 1, (len(pos), 3, 4))
    else:
        ctx.Shader.ObjectColor = (0.3, 0.7, 0.5, 1.0)
    ref = O.OracleContext(w, h)
    assert tuple(ctx.DrawMesh(mesh)) == ref.draw(mesh, ctx.state(), ctx.shader_struct())
    assert np.array_equal(ctx.Image(), ref.color())
    assert np.array_equal(ctx.DepthBuffer.view(np.uint64), ref.depth().view(np.uint64))
    return ctx.LastStats()


@pytest.mark.parametrize("vertex_colors", [False, True])
@pytest.mark.parametrize("n", [1, 33, 2048, 2049])
def test_clip_entries(gpu_lib, n, vertex_colors):
    rng = np.random.RandomState(n)
    pos = np.empty((n, 3, 3))
    pos[:, 0] = rng.uniform(-0.9, 0.9, (n, 3))
    far = rng.uniform(-3, 3, (n, 2, 3))
    far[np.arange(n), 0, rng.randint(0, 3, n)] = rng.choice([-1, 1], n) * rng.uniform(1.1, 3, n)
    pos[:, 1:] = far
    st = _compare(pos, 61, 47, vertex_colors)
    assert st["clipped"] == n


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 4097])
def test_row_start_tiles(gpu_lib, n):
    rng = np.random.RandomState(n)
    c = rng.uniform(-0.7, 0.7, (n, 1, 3))
    pos = c + rng.uniform(-1, 1, (n, 3, 3)) * np.array([0.05, 0.28, 0.1])
    st = _compare(np.clip(pos, -0.99, 0.99), 96, 80, False)
    assert st["clipped"] == 0
