"""Frames of different sizes drawn by several threads at once: their bands, and
so the shared memory that each launch asks for, differ. Every call succeeds and
gives the frame drawn alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(16, 16), (97, 61), (128, 128), (640, 97), (7680, 8), (20000, 2), (3, 20000)]


@pytest.mark.parametrize("precision", [0, 1])
def test_sizes_beside_each_other(gpu_lib, precision):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.context import NewContext
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.meshops import DeviceMesh
    from fauxgl_gb300.shader import NewPhongShader
    from fauxgl_gb300.shapes import sphere_positions

    pos = sphere_positions(3)
    mesh = DeviceMesh.upload(Mesh(pos, pos))

    def frame(ctx):
        ctx.ClearColorBufferWith(scenes.BACKGROUND)
        ctx.ClearDepthBuffer()
        ctx.DrawMesh(mesh)
        return ctx.Image()

    def context(w, h):
        ctx = NewContext(w, h)
        ctx.Precision = precision
        ctx.Shader = NewPhongShader(scenes.camera_matrix(w, h), scenes.LIGHT, scenes.EYE)
        ctx.Shader.ObjectColor = scenes.OBJECT_COLOR
        return ctx

    want = [frame(context(w, h)) for w, h in SIZES]
    errors = []

    def work(i):
        try:
            ctx = context(*SIZES[i])
            for _ in range(300):
                assert np.array_equal(frame(ctx), want[i])
        except BaseException as e:  # reported below
            errors.append("%s: %r" % (SIZES[i], e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(SIZES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
