"""Autotune leaves `window` alone, which shapes nothing: no trial of it is timed,
and none is adopted for the noise of its timing."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [3, 100])
def test_window_stays(gpu_lib, window):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.batch import Batch
    from fauxgl_gb300.context import NewContext
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.meshops import DeviceMesh
    from fauxgl_gb300.shader import NewPhongShader
    from fauxgl_gb300.shapes import sphere_positions

    pos = sphere_positions(2)
    mesh = DeviceMesh.upload(Mesh(pos, pos))
    ctx = NewContext(64, 48)
    ctx.Shader = NewPhongShader(scenes.camera_matrix(64, 48), scenes.LIGHT, scenes.EYE)
    for _ in range(4):
        batch = Batch()
        batch.SetTuning(window=window)
        batch.Add(ctx, mesh)
        best = batch.Autotune(repeats=1)
        assert best["window"] == window and batch.Tuning()["window"] == window
