"""Frames of a batch read back to overlapping places: copied in the order of the
items, so that the later one stays. Read-backs that are worth a second pass are
copied on two streams, in no order between them: where two of them overlap the
batch stays in one pass (as its launches show)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _render(at):
    """The kernel launches of one rendering."""
    import torch
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.batch import Batch
    from fauxgl_gb300.context import NewContext
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.meshops import DeviceMesh
    from fauxgl_gb300.shader import NewPhongShader
    from fauxgl_gb300.shapes import sphere_positions

    pos = sphere_positions(2)
    mesh = DeviceMesh.upload(Mesh(pos, pos))
    # four frames in the first pass, the small one and a fifth in the second:
    # the small one is ready for its copy while the first four are being copied
    sizes = [(3840, 2160)] * 4 + [(64, 48), (3840, 2160)]
    n, m = 3840 * 2160 * 4, 64 * 48 * 4
    out = torch.zeros(5 * n + m, dtype=torch.uint8, pin_memory=True)
    over = {"end": 4 * n - m, "start": 3 * n, "apart": 5 * n}[at]  # within the fourth frame, or not
    place = [0, n, 2 * n, 3 * n, over, 4 * n]

    class Overlapping(Batch):
        def _items(self):
            items = super()._items()
            for i, o in enumerate(place):
                items[i].out_nrgba = out.data_ptr() + o
            return items

    batch, ctxs = Overlapping(), []
    for w, h in sizes:
        ctx = NewContext(w, h)
        ctx.Shader = NewPhongShader(scenes.camera_matrix(w, h), scenes.LIGHT, scenes.EYE)
        ctx.Shader.ObjectColor = scenes.OBJECT_COLOR
        ctxs.append(ctx)
        batch.Add(ctx, mesh, read_back=True)
    for k in range(3):
        for i, ctx in enumerate(ctxs):
            ctx.ClearColorBufferWith((0.1 * k, 0.2, 0.1 * i, 1.0))
            ctx.ClearDepthBuffer()
        batch.Render()
        want = np.zeros(5 * n + m, np.uint8)
        for o, ctx in sorted(zip(place, ctxs), key=lambda p: p[1] is ctxs[4]):  # the small one last
            f = ctx.Image().ravel()
            want[o:o + len(f)] = f
        used = 5 * n + (m if at == "apart" else 0)
        assert np.array_equal(out.numpy()[:used], want[:used])
    return batch.LastStats()["kernel_launches"]


@pytest.mark.parametrize("at", ["end", "start"])
def test_later_read_back_stays(gpu_lib, at):
    assert _render(at) < _render("apart")
