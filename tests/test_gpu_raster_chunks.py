"""Chunks of the raster stage: several rounds of units with few fragments (most
pixels occluded), rounds whose fragments suddenly outgrow the estimate learnt
from the ones before (the chunk is redone), and pixels with many fragments in
one chunk, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _strips(rng, n, w, h, z, size):
    """n triangles of about `size` pixels at random places of a w x h frame, at depth z."""
    c = rng.uniform([-0.95, -0.95], [0.95, 0.95], (n, 1, 2))
    d = rng.uniform(-1, 1, (n, 3, 2)) * np.array([size / w, size / h]) * 2
    return np.concatenate([np.clip(c + d, -0.99, 0.99), np.broadcast_to(z, (n, 3))[..., None]], -1)


@pytest.mark.parametrize("order", ["hidden_first", "visible_first", "alternating", "stacked"])
@pytest.mark.parametrize("shader", ["solid", "phong", "blend"])
@pytest.mark.parametrize("w,h", [(200, 12), (4500, 3)])
def test_rounds_match_oracle(gpu_lib, order, shader, w, h):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.geom import Identity
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader, NewSolidColorShader
    from oracle import oracle as O

    rng = np.random.RandomState(7)
    n = 1500
    wall = np.array([[[-1, -1, 0.0], [1, -1, 0.0], [1, 1, 0.0]], [[-1, -1, 0.0], [1, 1, 0.0], [-1, 1, 0.0]]])
    hidden = _strips(rng, n, w, h, 0.5, 14)
    shown = _strips(rng, n, w, h, -0.5, 14)
    if order == "hidden_first":
        pos = np.concatenate([hidden, shown])
    elif order == "visible_first":
        pos = np.concatenate([shown, hidden])
    elif order == "alternating":
        pos = np.stack([hidden, shown], 1).reshape(-1, 3, 3)
    else:  # the same few places again and again, each nearer than the last
        pos = np.tile(_strips(rng, 6, w, h, 0.0, 20), (n // 6, 1, 1))
        pos[..., 2] = np.linspace(-0.01, -0.9, len(pos))[:, None]
    ctx = NewContext(w, h)
    ctx.Cull = CullNone
    ref = O.OracleContext(w, h)
    color = (0.3, 0.7, 0.5, 0.4 if shader == "blend" else 1.0)
    if shader == "solid" or shader == "blend":
        ctx.Shader = NewSolidColorShader(Identity(), color)
    else:
        ctx.Shader = NewPhongShader(Identity(), scenes.LIGHT, scenes.EYE)
        ctx.Shader.ObjectColor = color
    for m in (Mesh(wall, np.ones_like(wall)), Mesh(pos, rng.normal(size=pos.shape))):
        assert tuple(ctx.DrawMesh(m)) == ref.draw(m, ctx.state(), ctx.shader_struct())
    assert np.array_equal(ctx.Image(), ref.color())
    assert np.array_equal(ctx.DepthBuffer.view(np.uint64), ref.depth().view(np.uint64))
