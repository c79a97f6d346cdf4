"""The raster kernel's shared memory for any fragment cap a caller sets: its
layout and size on the CPU (rasterfit_check.cpp), and on the GPU frames drawn
with caps that are odd, or become odd when halved, against the oracle."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_layout_is_aligned_and_fits(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "rasterfit_check")
    subprocess.run([cxx, "-O2", "-std=c++17", os.path.join(HERE, "rasterfit_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [257, 767, 770, 1001, 4095, 2 ** 31 - 1])
@pytest.mark.parametrize("shader", ["solid", "phong", "mixed"])
@pytest.mark.parametrize("w,h", [(97, 61), (25900, 3)])
def test_any_fragment_cap_matches_oracle(gpu_lib, cap, shader, w, h):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.batch import Batch
    from fauxgl_gb300.context import PRECISION_MIXED, CullNone, NewContext
    from fauxgl_gb300.geom import Identity
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader, NewSolidColorShader
    from oracle import oracle as O

    rng = np.random.RandomState(w)
    small = rng.uniform(-0.9, 0.9, (300, 1, 3)) + rng.uniform(-1, 1, (300, 3, 3)) * np.array([10 / w, 10 / h, 0.05])
    large = rng.uniform(-0.95, 0.95, (30, 3, 3))  # rows of up to the frame's width: the span walk
    for pos in (np.clip(small, -0.99, 0.99), np.concatenate([np.clip(small, -0.99, 0.99), large])):
        mesh = Mesh(pos, rng.normal(size=pos.shape))
        ctx = NewContext(w, h)
        ctx.Cull = CullNone
        if shader == "solid":
            ctx.Shader = NewSolidColorShader(Identity(), (0.3, 0.7, 0.5, 0.4))
        else:
            ctx.Shader = NewPhongShader(Identity(), scenes.LIGHT, scenes.EYE)
            ctx.Shader.ObjectColor = scenes.OBJECT_COLOR
        if shader == "mixed":
            ctx.Precision = PRECISION_MIXED
        batch = Batch()
        batch.SetTuning(fragment_cap=cap)
        batch.Add(ctx, mesh)
        ref = O.OracleContext(w, h)
        assert tuple(batch.Render()[0]) == ref.draw(mesh, ctx.state(), ctx.shader_struct())
        assert np.array_equal(ctx.DepthBuffer.view(np.uint64), ref.depth().view(np.uint64))
        step = np.abs(ctx.Image().astype(int) - ref.color().astype(int)).max()
        assert step <= (1 if shader == "mixed" else 0)  # one step in the mixed form


@pytest.mark.gpu
@pytest.mark.parametrize("cap,widest", [(256, 26028), (257, 26844), (300, 26703), (1000, 26104), (1024, 26028)])
def test_widest_frame_of_a_cap(gpu_lib, cap, widest):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300._abi import FauxGLError
    from fauxgl_gb300.batch import Batch
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.geom import Identity
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader
    from oracle import oracle as O

    rng = np.random.RandomState(cap)
    pos = rng.uniform(-0.95, 0.95, (200, 1, 3)) + rng.uniform(-1, 1, (200, 3, 3)) * np.array([2e-3, 0.9, 0.02])
    pos[150:] = rng.uniform(-0.95, 0.95, (50, 3, 3))
    mesh = Mesh(np.clip(pos, -0.99, 0.99), rng.normal(size=pos.shape), None, rng.uniform(0, 1, (200, 3, 4)))
    for w in (widest, widest + 1):
        ctx = NewContext(w, 2)
        ctx.Cull = CullNone
        ctx.Shader = NewPhongShader(Identity(), scenes.LIGHT, scenes.EYE)
        batch = Batch()
        batch.SetTuning(fragment_cap=cap)
        batch.Add(ctx, mesh)
        if w > widest:
            with pytest.raises(FauxGLError):
                batch.Render()
            continue
        ref = O.OracleContext(w, 2)
        assert tuple(batch.Render()[0]) == ref.draw(mesh, ctx.state(), ctx.shader_struct())
        assert np.array_equal(ctx.Image(), ref.color())
        assert np.array_equal(ctx.DepthBuffer.view(np.uint64), ref.depth().view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,band,accepted", [(320, 180, 26027, True), (320, 180, 26240, False), (320, 180, 31000, False),
                                               (320, 80, 60000, True), (160, 200, 60000, True), (700, 100, 66000, False)])
def test_band_size_of_the_tuning(gpu_lib, w, h, band, accepted):
    """A band of band_pixels (whole rows, at most 128) has to fit, though small passes take smaller ones."""
    from fauxgl_gb300 import scenes
    from fauxgl_gb300._abi import FauxGLError
    from fauxgl_gb300.batch import Batch
    from fauxgl_gb300.context import NewContext
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader
    from fauxgl_gb300.shapes import sphere_positions

    pos = sphere_positions(2)
    ctx = NewContext(w, h)
    ctx.Shader = NewPhongShader(scenes.camera_matrix(w, h), scenes.LIGHT, scenes.EYE)
    batch = Batch()
    batch.SetTuning(band_pixels=band)
    batch.Add(ctx, Mesh(pos, pos))
    if not accepted:
        with pytest.raises(FauxGLError):
            batch.Render()
        return
    total = batch.Render()[0].TotalPixels
    alone = NewContext(w, h)
    alone.Shader = ctx.Shader
    assert alone.DrawMesh(Mesh(pos, pos)).TotalPixels == total > 0
    assert np.array_equal(alone.Image(), ctx.Image())
