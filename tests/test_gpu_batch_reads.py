"""Batches whose read-backs are worth a second pass (the first frames are then
copied beside it), against the same draws on their own: full-size and
downsampled read-backs in one batch, draws without one, a frame drawn twice
(read after its last draw), and buffers that have to grow on the first run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "scaled", "some", "twice", "grow"])
@pytest.mark.parametrize("n", [35, 36, 41])
def test_batch_reads_match_single_draws(gpu_lib, form, n):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.batch import Batch
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.geom import Identity
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.meshops import DeviceMesh
    from fauxgl_gb300.shader import NewPhongShader

    rng = np.random.RandomState(n)
    tris = 4000 if form == "grow" else 60
    meshes = []
    for _ in range(3):
        pos = rng.uniform(-1.4, 1.4, (tris, 3, 3))
        meshes.append(DeviceMesh.upload(Mesh(pos, rng.normal(size=pos.shape))))

    def context(i, w, h):
        ctx = NewContext(w, h)
        ctx.Cull = CullNone
        ctx.ClearColorBufferWith((0.1, 0.2, 0.01 * (i % 7), 1.0))
        ctx.ClearDepthBuffer()
        ctx.Shader = NewPhongShader(Identity(), scenes.LIGHT, scenes.EYE)
        ctx.Shader.ObjectColor = (0.3, 0.7, 0.02 * (i % 9), 1.0)
        return ctx

    batch, want = Batch(), []
    last = {}
    for i in range(n):
        w, h = 24 + 2 * (i % 5), 16 + 4 * (i % 3)
        scale = 2 if form == "scaled" and i % 3 == 0 else 1
        read = not (form == "some" and i % 4 == 1)
        if form == "twice" and i % 6 == 5:
            ctx, single = last["pair"]
        else:
            ctx, single = context(i, w, h), context(i, w, h)
        last["pair"] = (ctx, single)
        mesh = meshes[i % 3]
        batch.Add(ctx, mesh, read_back=read, scale=scale)
        info = single.DrawMesh(mesh)
        want.append((single, info, read, scale))
    infos = batch.Render()
    for i, (single, info, read, scale) in enumerate(want):
        assert tuple(infos[i]) == tuple(info)
        if read:
            assert np.array_equal(batch.Result(i), single.Image() if scale == 1 else single.Downsample(scale)), i
