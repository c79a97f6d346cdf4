"""Passes that mix draws whose plain-form colours are certified in FP32 with draws
shaded in FP64 (their fragment records differ in size), and bands with more
uncertain fragments than the pending list holds, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 1, 2])
def test_certified_beside_fp64_draws(gpu_lib, order):
    from fauxgl_gb300 import NewImageTexture, scenes
    from fauxgl_gb300.batch import Batch
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader, NewSolidColorShader, NewTextureShader
    from fauxgl_gb300.shapes import sphere_positions
    from oracle import oracle as O

    rng = np.random.RandomState(order)
    batch, want = Batch(), []
    kinds = ["object", "texture", "vertex", "solid", "textured phong", "power", "object", "clipped"]
    for i, kind in enumerate(np.roll(kinds, order * 3)):
        w, h = [(97, 61), (300, 20), (33, 150), (640, 97)][(i + order) % 4]
        pos = scenes.displace(sphere_positions(1 + i % 4), i)
        if kind == "clipped":
            pos = pos * 6
        n = len(pos)
        mesh = Mesh(pos, pos, rng.uniform(-0.5, 1.5, (n, 3, 2)), rng.uniform(0, 1, (n, 3, 4)))
        texture = NewImageTexture(rng.randint(0, 65536, (5, 9, 4)).astype(np.uint16))
        ctx = NewContext(w, h)
        ctx.Cull = CullNone
        ctx.ClearColorBufferWith(scenes.BACKGROUND)
        matrix = scenes.camera_matrix(w, h)
        tex = None
        if kind == "texture":
            ctx.Shader, tex = NewTextureShader(matrix, texture), texture
        elif kind == "solid":
            ctx.Shader = NewSolidColorShader(matrix, (0.2, 0.9, 0.4, 0.5))
        else:
            ctx.Shader = NewPhongShader(matrix, scenes.LIGHT, scenes.EYE)
            if kind != "vertex":
                ctx.Shader.ObjectColor = (0.3, 0.7, 0.5, 1.0)
            if kind == "power":
                ctx.Shader.SpecularPower = 7.5
            if kind == "textured phong":
                ctx.Shader.Texture, tex = texture, texture
        batch.Add(ctx, mesh)
        ref = O.OracleContext(w, h)
        ref.clear_color(scenes.BACKGROUND)
        want.append((ctx, ref, ref.draw(mesh, ctx.state(), ctx.shader_struct(), texture=tex), kind))
    for info, (ctx, ref, ref_info, kind) in zip(batch.Render(), want):
        assert tuple(info) == ref_info, kind
        assert np.array_equal(ctx.Image(), ref.color()), kind
        assert np.array_equal(ctx.DepthBuffer.view(np.uint64), ref.depth().view(np.uint64)), kind


@pytest.mark.parametrize("w,h", [(4099, 3), (9001, 2), (1030, 40)])
@pytest.mark.parametrize("order", ["back to front", "front to back", "mixed"])
def test_pending_list_overflows(gpu_lib, w, h, order):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.geom import Identity
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader
    from oracle import oracle as O

    rng = np.random.RandomState(w)
    # layers over the whole frame and small triangles between them; an ambient
    # light of 1 and a colour of k / 255 put every fragment on a byte's boundary
    layers = np.linspace(0.8, -0.8, 6)
    pos = []
    for k, z in enumerate(layers):
        a, b = 0.9, 0.99 - 0.02 * k
        pos += [[[-b, -a, z], [b, -a, z], [b, a, z - 0.01]], [[-b, -a, z], [b, a, z - 0.01], [-b, a, z]]]
        c = rng.uniform(-0.95, 0.95, (60, 1, 3)) * [1, 1, 0] + [0, 0, z - 0.1]
        pos += list(np.clip(c + rng.uniform(-1, 1, (60, 3, 3)) * [8 / w, 4 / h, 0.1], -0.99, 0.99))
    pos = np.array(pos)
    if order == "front to back":
        pos = pos[::-1].copy()
    elif order == "mixed":
        pos = pos[rng.permutation(len(pos))]
    mesh = Mesh(pos, rng.normal(size=pos.shape))
    ctx = NewContext(w, h)
    ctx.Cull = CullNone
    ctx.Shader = NewPhongShader(Identity(), scenes.LIGHT, scenes.EYE)
    ctx.Shader.ObjectColor = (100 / 255, 50 / 255, 200 / 255, 1.0)
    ctx.Shader.AmbientColor = (1.0, 1.0, 1.0, 1.0)
    ctx.Shader.DiffuseColor = ctx.Shader.SpecularColor = (0.0, 0.0, 0.0, 1.0)
    ref = O.OracleContext(w, h)
    for lit in (False, True):  # the second draw over the first, with colours of its own
        if lit:
            ctx.Shader.DiffuseColor = (0.3, 0.2, 0.1, 1.0)
        assert tuple(ctx.DrawMesh(mesh)) == ref.draw(mesh, ctx.state(), ctx.shader_struct())
        assert np.array_equal(ctx.Image(), ref.color())
        assert np.array_equal(ctx.DepthBuffer.view(np.uint64), ref.depth().view(np.uint64))
