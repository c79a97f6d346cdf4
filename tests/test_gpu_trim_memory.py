"""Device memory is given back: when the last object is released all but 128 MiB of
each of the three pools, and everything unused on TrimMemory, also while other
objects live. A process of its own, so that no other test's objects live."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import numpy as np, torch
from fauxgl_gb300 import scenes
from fauxgl_gb300.context import NewContext
from fauxgl_gb300.mesh import Mesh
from fauxgl_gb300.meshops import DeviceMesh
from fauxgl_gb300.shader import NewPhongShader
MB = 1 << 20

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]

def context():
    c = NewContext(1280, 720)
    c.Shader = NewPhongShader(scenes.camera_matrix(1280, 720), scenes.LIGHT, scenes.EYE)
    c.Shader.ObjectColor = scenes.OBJECT_COLOR
    return c

def work(triangles):
    p = np.random.RandomState(1).randint(0, 1 << 11, (triangles, 3, 3)) / 1024.0 - 1.0
    c, d = context(), DeviceMesh.upload(Mesh(p, p))
    d.SmoothNormalsThreshold(0.5)
    lines = d.SharpEdges(0.5)
    if triangles <= 1000:
        c.DrawMesh(d)
    return c, d, lines

kept = work(1000)  # every kernel is loaded
image = kept[0].Image()
if TRIM:
    from fauxgl_gb300 import TrimMemory
    kept = None
    TrimMemory()
base = free()
for _ in range(2):
    kept = work(2000000)
    kept = None
left = (base - free()) / MB
assert left < 3 * 128 + 64, "kept %.0f MB after the last release" % left
if TRIM:
    TrimMemory()
    left = (base - free()) / MB
    assert left < 32, "kept %.0f MB after TrimMemory" % left
    live = context()
    live.DrawMesh(Mesh(np.eye(3)[None], np.eye(3)[None]))
    TrimMemory()
    before, want = free(), live.Image()
    kept = work(2000000)
    kept = None
    assert before - free() > 128 * MB  # kept for later calls
    TrimMemory()
    left = (before - free()) / MB
    assert left < 32, "kept %.0f MB beside a context" % left
    assert np.array_equal(live.Image(), want)
    live.DrawMesh(DeviceMesh.upload(Mesh(np.eye(3)[None], np.eye(3)[None])))  # and on it goes
    assert np.array_equal(work(1000)[0].Image(), image)
print("ok")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("trim", [False, True])
def test_memory_is_given_back(gpu_lib, trim):
    r = subprocess.run([sys.executable, "-c", SCRIPT.replace("if TRIM:", "if %s:" % trim)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
