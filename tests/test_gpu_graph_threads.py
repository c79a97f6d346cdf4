"""Batches issued as graphs in one thread while others make and release contexts,
meshes and textures: nothing that waits for the device or gives memory back may
fall into a capture. Every call succeeds and every frame is the one drawn alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["contexts", "growing", "meshes", "textures", "all"])
def test_captures_beside_other_threads(gpu_lib, what):
    from fauxgl_gb300 import NewImageTexture, scenes
    from fauxgl_gb300.batch import Batch
    from fauxgl_gb300.context import NewContext
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.meshops import DeviceMesh
    from fauxgl_gb300.shader import NewPhongShader, NewTextureShader
    from fauxgl_gb300.shapes import sphere_positions

    spheres = [Mesh(p, p) for p in (sphere_positions(d) for d in (1, 3))]
    mesh = DeviceMesh.upload(spheres[1])
    image = np.random.RandomState(1).randint(0, 65536, (9, 7, 4)).astype(np.uint16)

    def context(w, h):
        c = NewContext(w, h)
        c.ClearColorBufferWith(scenes.BACKGROUND)
        c.Shader = NewPhongShader(scenes.camera_matrix(w, h), scenes.LIGHT, scenes.EYE)
        c.Shader.ObjectColor = scenes.OBJECT_COLOR
        return c

    def contexts(k):
        c = context(40 + k % 50, 40)
        c.DrawMesh(mesh)
        return c.Image()

    def growing(k):
        c = context(64, 64)
        for m in spheres:
            c.DrawMesh(DeviceMesh.upload(m))
        return c.Image()

    def meshes(k):
        d = DeviceMesh.upload(spheres[1])
        d.SmoothNormals()
        return d.download().tri_nrm

    def textures(k):
        c = context(50, 40)
        tex = Mesh(spheres[0].tri_pos, spheres[0].tri_nrm, spheres[0].tri_pos[..., :2].copy())
        c.Shader = NewTextureShader(c.Shader.Matrix, NewImageTexture(image))
        c.DrawMesh(tex)
        return c.Image()

    jobs = {"contexts": contexts, "growing": growing, "meshes": meshes, "textures": textures}
    if what != "all":
        jobs = {what: jobs[what]}
    want = {name: [job(k) for k in range(50)] for name, job in jobs.items()}
    sizes = [(64 + 8 * i, 48) for i in range(6)]
    frames = []
    for w, h in sizes:
        c = context(w, h)
        c.DrawMesh(mesh)
        frames.append(c.Image())
    errors = []
    done = threading.Event()

    def draw():
        batch = Batch(use_graph=True)
        targets = [context(*s) for s in sizes]
        for _ in range(400):
            batch.Clear()
            for c in targets:
                c.ClearColorBufferWith(scenes.BACKGROUND)
                c.ClearDepthBuffer()
                batch.Add(c, mesh, read_back=True)
            batch.Render()
            for i, f in enumerate(frames):
                assert np.array_equal(batch.Result(i), f)

    def other(name):
        k = 0
        while not done.is_set() and k < 20000:
            assert np.array_equal(jobs[name](k), want[name][k % 50], equal_nan=name == "meshes")
            k += 1
        assert k > 0

    def run(f, *args):
        try:
            f(*args)
        except BaseException as e:  # reported below
            errors.append("%s%s: %r" % (f.__name__, args, e))
        finally:
            if f is draw:
                done.set()

    threads = [threading.Thread(target=run, args=(draw,))]
    threads += [threading.Thread(target=run, args=(other, name)) for name in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
