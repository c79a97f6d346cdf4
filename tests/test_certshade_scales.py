"""cert_shade (fgc_certshade.cuh) at the ends of FP32's range: on the CPU against
an FP64 evaluation over magnitudes from the whole exponent range
(certshade_scales_check.cpp), and on the GPU frames of meshes whose normals, or
which themselves, are very small, against the oracle."""
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
    exe = str(tmp_path / "certshade_scales_check")
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-std=c++17", os.path.join(HERE, "certshade_scales_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe, "3000000"], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("colors", [False, True])
@pytest.mark.parametrize("normal,scene", [(1e-12, 1.0), (1e-19, 1.0), (1e-21, 1.0), (1e-40, 1.0), (1e25, 1.0),
                                          (1.0, 1e-19), (1.0, 1e-21), (1e-20, 1e-20)])
def test_small_vectors_match_oracle(gpu_lib, normal, scene, colors):
    from fauxgl_gb300 import scenes
    from fauxgl_gb300.context import CullNone, NewContext
    from fauxgl_gb300.geom import Scale, V
    from fauxgl_gb300.mesh import Mesh
    from fauxgl_gb300.shader import NewPhongShader
    from fauxgl_gb300.shapes import sphere_positions
    from oracle import oracle as O

    pos = scenes.displace(sphere_positions(4), 5)
    col = None
    if colors:
        col = np.random.RandomState(2).uniform(0, 1, (len(pos), 3, 4))
        col[..., 3] = 1.0
    mesh = Mesh(pos * scene, pos * normal, None, col)
    w, h = 320, 200
    ctx = NewContext(w, h)
    ctx.Cull = CullNone
    ctx.ClearColorBufferWith(scenes.BACKGROUND)
    matrix = scenes.camera_matrix(w, h).Mul(Scale(V(1 / scene, 1 / scene, 1 / scene)))
    eye = np.asarray([scenes.EYE.X, scenes.EYE.Y, scenes.EYE.Z]) * scene
    ctx.Shader = NewPhongShader(matrix, scenes.LIGHT, V(*eye))
    if not colors:
        ctx.Shader.ObjectColor = scenes.OBJECT_COLOR
    ref = O.OracleContext(w, h)
    ref.clear_color(scenes.BACKGROUND)
    assert tuple(ctx.DrawMesh(mesh)) == ref.draw(mesh, ctx.state(), ctx.shader_struct())
    assert np.array_equal(ctx.Image(), ref.color())
