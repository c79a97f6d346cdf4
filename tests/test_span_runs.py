"""Wide primitives: triangles of many widths, whose rows begin and end at every
place of the raster stage's runs, against the oracle."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(33, 40), (64, 9), (257, 130), (1023, 77), (4099, 5)])
@pytest.mark.parametrize("precision", [0, 1])
def test_wide_triangles_match_oracle(gpu_lib, w, h, precision):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.geom import Identity
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader
    from oracle import oracle as O

    rng = np.random.RandomState(w * 7 + h)
    n = 60
    pos = rng.uniform(-1.3, 1.3, (n, 3, 3))  # some reach beyond the frame and are clipped
    pos[: n // 2] = rng.uniform(-0.95, 0.95, (n // 2, 3, 3))
    pos[:10, :, 0] = np.round(pos[:10, :, 0] * w) / w  # corners on pixel edges
    pos[10:20, 1, 1] = pos[10:20, 0, 1]                # horizontal edges
    pos[20:26, :, 1] = pos[20:26, :1, 1] + rng.uniform(-1, 1, (6, 3)) * 1.5 / h  # slivers a row or two tall
    mesh = Mesh(pos, rng.normal(size=(n, 3, 3)))
    ctx = NewContext(w, h)
    ctx.Cull = CullNone
    ctx.Precision = precision
    sh = NewPhongShader(Identity(), scenes.LIGHT, scenes.EYE)
    sh.ObjectColor = scenes.OBJECT_COLOR
    ctx.Shader = sh
    ref = O.OracleContext(w, h)
    assert tuple(ctx.DrawMesh(mesh)) == ref.draw(mesh, ctx.state(), ctx.shader_struct())
    assert np.array_equal(ctx.DepthBuffer.view(np.uint64), ref.depth().view(np.uint64))
    d = np.abs(ctx.Image().astype(int) - ref.color().astype(int)).max()
    assert d <= precision  # one step in the mixed form, none in the plain one
