"""Texture sampling where it takes another path: coordinates outside [0, 1), at
0 and 1 and on texels, textures with and without alpha, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coords", ["inside", "outside", "corners", "texels"])
@pytest.mark.parametrize("alpha", ["opaque", "mixed"])
@pytest.mark.parametrize("size", [(1, 1), (2, 3), (17, 8)])
def test_texture_coordinates(gpu_lib, coords, alpha, size):
    from fauxgl_gb300 import NewImageTexture
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.geom import Identity
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewTextureShader
    from oracle import oracle as O

    rng = np.random.RandomState(3)
    w, h = size
    im = rng.randint(0, 256, (h, w, 4)).astype(np.uint8)
    if alpha == "opaque":
        im[..., 3] = 255
    n = 40
    pos = rng.uniform(-0.95, 0.95, (n, 3, 3))
    tex = rng.uniform(0, 1, (n, 3, 2))
    if coords == "outside":
        tex = rng.uniform(-2.5, 3.5, (n, 3, 2))
    elif coords == "corners":
        tex = rng.randint(-1, 3, (n, 3, 2)).astype(float)
    elif coords == "texels":
        tex = np.broadcast_to(rng.randint(0, 3, (n, 1, 2)) / np.array([max(w - 1, 1), max(h - 1, 1)]), (n, 3, 2)).copy()
    mesh = Mesh(pos, np.ones_like(pos), tex)
    ctx = NewContext(70, 50)
    ctx.Cull = CullNone
    texture = NewImageTexture(im.astype(np.uint16) * 257)
    ctx.Shader = NewTextureShader(Identity(), texture)
    ref = O.OracleContext(70, 50)
    assert tuple(ctx.DrawMesh(mesh)) == ref.draw(mesh, ctx.state(), ctx.shader_struct(), texture=texture)
    assert np.array_equal(ctx.Image(), ref.color())
