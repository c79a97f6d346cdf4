"""cert_shade (fgc_certshade.cuh), the FP32 interval form of PhongShader's
colour bytes: on the CPU against an FP64 evaluation over random and edge
inputs (certshade_check.cpp), and on the GPU whole frames against the oracle
where certification is at its limits."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_certified_bytes_match_fp64(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "certshade_check")
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-std=c++17", os.path.join(HERE, "certshade_check.cpp"), "-o",
                    exe], check=True)
    r = subprocess.run([exe, "1000000"], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


# power, ambient, diffuse, specular, colour, flat normals, alpha blending off with alpha < 1
CASES = {
    "default": (32.0, 0.2, 0.8, 1.0, (70 / 255, 137 / 255, 102 / 255, 1.0), False),
    # whole faces on a byte boundary: lights of k/255 steps and a flat mesh, every fragment goes to the pending list
    "boundary": (32.0, 0.0, 0.0, 0.0, (0.5, 0.5, 0.5, 1.0), True),
    "boundary_lit": (32.0, 1.0, 0.0, 0.0, (100 / 255, 50 / 255, 200 / 255, 1.0), False),
    "highlight": (2.0, 0.0, 0.1, 3.0, (0.9, 0.8, 1.0, 1.0), False),
    "steep": (128.0, 0.2, 0.8, 1.0, (1.0, 1.0, 1.0, 1.0), False),
    "beyond_power": (129.0, 0.2, 0.8, 1.0, (1.0, 1.0, 1.0, 1.0), False),
    "fractional_power": (2.5, 0.2, 0.8, 0.0, (0.3, 0.6, 0.9, 1.0), False),
    "negative_diffuse": (32.0, 0.6, -0.5, 1.0, (0.3, 0.6, 0.9, 1.0), False),
    "see_through": (32.0, 0.2, 0.8, 1.0, (0.3, 0.6, 0.9, 0.5), False),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("size,detail", [((97, 61), 3), ((640, 97), 2), ((1500, 40), 5)])
def test_frames_match_oracle(gpu_lib, name, size, detail):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader
    from fauxgl_gb300.shapes import sphere_positions, _with_face_normals
    from oracle import oracle as O

    power, amb, dif, spec, color, flat = CASES[name]
    pos = scenes.displace(sphere_positions(detail), 5)
    mesh = _with_face_normals(pos) if flat else Mesh(pos, pos)
    w, h = size
    ctx = NewContext(w, h)
    ctx.Cull = CullNone
    ctx.ClearColorBufferWith(scenes.BACKGROUND)
    sh = NewPhongShader(scenes.camera_matrix(w, h), scenes.LIGHT, scenes.EYE)
    sh.ObjectColor = color
    sh.AmbientColor, sh.DiffuseColor, sh.SpecularColor = (amb,) * 3 + (1,), (dif,) * 3 + (1,), (spec,) * 3 + (1,)
    sh.SpecularPower = power
    ctx.Shader = sh
    ref = O.OracleContext(w, h)
    ref.clear_color(scenes.BACKGROUND)
    for draw in range(2):  # the second over the first's colours and depth
        info = ctx.DrawMesh(mesh)
        assert tuple(info) == ref.draw(mesh, ctx.state(), ctx.shader_struct())
    assert np.array_equal(ctx.Image(), ref.color())
    assert np.array_equal(ctx.DepthBuffer.view(np.uint64), ref.depth().view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("blend", [True, False])
@pytest.mark.parametrize("colors", ["opaque", "alphas", "zeros", "wild", "boundary"])
@pytest.mark.parametrize("size,detail", [((97, 61), 3), ((640, 97), 2), ((1500, 40), 5)])
def test_vertex_colors_match_oracle(gpu_lib, colors, blend, size, detail):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader
    from fauxgl_gb300.shapes import sphere_positions
    from oracle import oracle as O

    pos = scenes.displace(sphere_positions(detail), 5)
    n = len(pos)
    rng = np.random.RandomState(2)
    col = rng.uniform(0, 1, (n, 3, 4))
    col[..., 3] = 1.0
    if colors == "alphas":
        col[..., 3] = rng.choice([0.0, 0.3, 1.0, 1.5], (n, 3))
    elif colors == "zeros":
        col[rng.uniform(size=n) < 0.5] = 0.0
    elif colors == "wild":
        col[..., :3] = rng.choice([-0.5, 0.0, 1e-20, 1.0, 3.0, 1e9], (n, 3, 3))
    elif colors == "boundary":  # whole faces of k / 255 steps
        col[..., :3] = rng.randint(0, 256, (n, 1, 3)) / 255.0
    mesh = Mesh(pos, pos, None, col)
    w, h = size
    ctx = NewContext(w, h)
    ctx.Cull = CullNone
    ctx.AlphaBlend = blend
    ctx.ClearColorBufferWith(scenes.BACKGROUND)
    eye = scenes.EYE
    ctx.Shader = NewPhongShader(scenes.camera_matrix(w, h), scenes.LIGHT, eye)
    ref = O.OracleContext(w, h)
    ref.clear_color(scenes.BACKGROUND)
    for draw in range(2):
        info = ctx.DrawMesh(mesh)
        assert tuple(info) == ref.draw(mesh, ctx.state(), ctx.shader_struct())
    assert np.array_equal(ctx.Image(), ref.color())
    assert np.array_equal(ctx.DepthBuffer.view(np.uint64), ref.depth().view(np.uint64))
