"""The workloads this framework's speed is judged on.

Each case is work a program that draws with this package has it do, through the public API:
frames through Context (clear, DrawMesh, Image), supersampled frames with an overlay and a
box downsample, feature lines, batches of thumbnails, meshes drawn straight from host arrays,
and mesh preparation from an STL file. Meshes are displaced icospheres and lathe shapes of the
sizes that the benchmark, the serving pool and the tests use; every input follows from the
case and the seed. A case's "kind" says which of these it is:

  frame     Clear, DrawMesh, Image (and, where "depth", DepthBuffer)
  overlay   a frame at "scale" times the size, a wireframe overlay, Downsample(scale)
  lines     a frame, then the mesh's sharp edges and silhouette found anew and drawn over it
  batch     "views" thumbnails of several meshes, one Batch, every frame read back
  prepare   LoadSTL of a binary file in memory, SmoothNormalsThreshold, read back
"""
import math
import struct

import numpy as np
import torch

from fauxgl_gb300 import NewImageTexture, scenes
from fauxgl_gb300.batch import Batch
from fauxgl_gb300.context import PRECISION_MIXED, PRECISION_PLAIN, NewContext
from fauxgl_gb300.geom import Color, Radians, V, Vector
from fauxgl_gb300.mesh import Mesh
from fauxgl_gb300.meshops import DeviceMesh
from fauxgl_gb300.shader import NewPhongShader, NewSolidColorShader, NewTextureShader
from fauxgl_gb300.shapes import cylinder_segments, sphere_positions

FAR = 1.0  # the depth of the far plane on the screen


def listed():
    return [
        # an icon or a preview: the smallest call, launches and host work decide
        dict(name="icon", kind="frame", mesh="sphere", detail=2, width=128, height=128, shader="phong",
             precision="plain", resident=True, depth=True),
        # the smallest benchmark scene: 5,120 triangles, its depth buffer read as well
        dict(name="sphere_512", kind="frame", mesh="sphere", detail=4, width=512, height=512, shader="phong",
             precision="plain", resident=True, depth=True),
        # the headline workload: 1.31 million triangles at 1080p, FP64 throughout
        dict(name="dense_1080p", kind="frame", mesh="sphere", detail=8, width=1920, height=1080, shader="phong",
             precision="plain", resident=True, depth=False),
        # the same frame in the mixed form (FP32 shading)
        dict(name="dense_1080p_mixed", kind="frame", mesh="sphere", detail=8, width=1920, height=1080,
             shader="phong", precision="mixed", resident=True, depth=False),
        # a textured model at an ordinary size
        dict(name="textured_720p", kind="frame", mesh="sphere", detail=6, width=1280, height=720, shader="texture",
             precision="plain", resident=True, depth=False),
        # a few hundred triangles seen from close by: large, clipped triangles and long rows at an odd size
        dict(name="closeup_1079", kind="frame", mesh="lathe", detail=96, width=1919, height=1079, shader="phong",
             precision="plain", resident=True, depth=False),
        # a program that edits its mesh: host arrays with vertex colours drawn once, nothing kept on the device
        dict(name="edited_mesh_720p", kind="frame", mesh="sphere", detail=6, width=1280, height=720,
             shader="vertex", precision="plain", resident=False, depth=False),
        # the largest call: 16 samples per pixel, a wireframe overlay, the box downsample
        dict(name="supersampled_overlay", kind="overlay", mesh="sphere", detail=8, width=1920, height=1080, scale=4,
             precision="plain"),
        # a model with its feature lines found for this view and drawn over it
        dict(name="feature_lines_900p", kind="lines", mesh="sphere", detail=7, width=1600, height=900,
             precision="plain"),
        # a page of thumbnails in one submission, mixed form
        dict(name="thumbnails_mixed", kind="batch", views=48, scale=1, precision="mixed"),
        # fewer, with 2 x 2 samples per pixel, FP64
        dict(name="thumbnails_ss2_plain", kind="batch", views=20, scale=2, precision="plain"),
        # a 16 MB binary STL to a smoothed mesh in host arrays
        dict(name="stl_to_smooth", kind="prepare", detail=7, degrees=30),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "frame", "overlay", "lines", "batch", "batch", "prepare"])
    precision = rng.choice(["plain", "plain", "mixed"])
    if kind == "frame":
        lathe = rng.random() < 0.25
        resident = rng.random() < 0.75
        detail = _log(rng, 8, 512) if lathe else rng.randint(2, 8 if resident else 7)
        width, height = _log(rng, 128, 1920), _log(rng, 128, 1080)
        return dict(kind=kind, mesh="lathe" if lathe else "sphere", detail=detail, width=width, height=height,
                    shader="phong" if lathe else rng.choice(["phong", "phong", "texture", "vertex"]),
                    precision=precision, resident=resident, depth=width * height <= 1 << 18 and not lathe and detail <= 5)
    if kind == "overlay":
        scale = rng.choice([2, 4])
        return dict(kind=kind, mesh="sphere", detail=rng.randint(5, 8), width=_log(rng, 480, 1920),
                    height=_log(rng, 270, 1080), scale=scale, precision=precision)
    if kind == "lines":
        return dict(kind=kind, mesh="sphere", detail=rng.randint(4, 8), width=_log(rng, 320, 1920),
                    height=_log(rng, 200, 1080), precision=precision)
    if kind == "batch":
        scale = rng.choice([1, 2])
        return dict(kind=kind, views=rng.randint(3, 48 if scale == 1 else 20), scale=scale, precision=precision)
    return dict(kind=kind, detail=rng.randint(4, 7), degrees=rng.randint(15, 60))


# -- inputs -------------------------------------------------------------------
_spheres = {}


def _sphere(detail):
    """The unit icosphere's corners on the GPU, (T, 3, 3)."""
    if detail not in _spheres:
        _spheres[detail] = torch.from_numpy(sphere_positions(detail)).cuda()
    return _spheres[detail]


def _rng(case, seed):
    return np.random.RandomState((seed * 7919 + len(case)) % (1 << 32))


def _displaced(detail, rng):
    """Corner positions of a displaced icosphere (8 sine octaves, as the benchmark's meshes), fit
    to the bi-unit cube, and its face normals: (T, 3, 3) and (T, 3) on the GPU. Equal corners
    stay equal: every operation is elementwise."""
    p = _sphere(detail)
    r = torch.ones_like(p[..., 0])
    for k in range(8):
        d = rng.normal(size=3)
        d *= 3.0 * 2.0 ** k / np.linalg.norm(d)
        r += 0.15 * 2.0 ** -k * torch.sin(d[0] * p[..., 0] + d[1] * p[..., 1] + d[2] * p[..., 2]
                                          + 2 * math.pi * rng.uniform())
    p = p * r[..., None]
    lo, hi = p.amin((0, 1)), p.amax((0, 1))
    p = (p - (lo + hi) / 2) * (2.0 / (hi - lo).max())
    n = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    return p.contiguous(), n / n.norm(dim=1, keepdim=True)


def _sphere_mesh(case, rng):
    """A host Mesh of the displaced sphere with face normals, texture coordinates and colours as
    the case's shader reads them."""
    p, n = _displaced(case["detail"], rng)
    nrm = n[:, None, :].expand(-1, 3, -1).contiguous()
    tex = col = None
    if case.get("shader") == "texture":
        u = _sphere(case["detail"])
        tex = torch.stack([torch.atan2(u[..., 0], u[..., 2]) / (2 * math.pi) + 0.5,
                           torch.asin(u[..., 1].clamp(-1, 1)) / math.pi + 0.5], -1).cpu().numpy()
    if case.get("shader") == "vertex":
        c = (p * 0.5 + 0.5).clamp(0, 1)
        col = torch.cat([c, torch.ones_like(c[..., :1])], -1).cpu().numpy()
    return Mesh(p.cpu().numpy(), nrm.cpu().numpy(), tex, col)


def _smoothed(mesh):
    """The mesh on the device with its normals smoothed at 30 degrees, as the examples prepare it."""
    d = DeviceMesh.upload(mesh)
    d.SmoothNormalsThreshold(Radians(30.0))
    return d


def _lathe_mesh(segments, rng):
    m = cylinder_segments(segments, capped=True, cone=rng.uniform() < 0.3)
    m.BiUnitCube()
    return m


def _texture(rng):
    """A 512 x 256 image of smooth noise with a checker over it."""
    y, x = np.mgrid[0:256, 0:512]
    img = np.full((256, 512, 4), 255, dtype=np.uint32)
    for c in range(3):
        f, g, a = rng.uniform(0.01, 0.08), rng.uniform(0.01, 0.08), rng.uniform(0, 6)
        img[..., c] = 128 + 100 * np.sin(f * x + g * y + a) + 20 * ((x // 16 + y // 16) % 2)
    return NewImageTexture((img * 257).astype(np.uint16))


def _eye(rng, radius):
    az, el = 2 * math.pi * rng.uniform(), math.radians(rng.uniform(-25, 35))
    return Vector(radius * math.cos(el) * math.cos(az), radius * math.sin(el), radius * math.cos(el) * math.sin(az))


def _phong(matrix, eye, color):
    sh = NewPhongShader(matrix, scenes.LIGHT, eye)
    if color is not None:
        sh.ObjectColor = color
    return sh


def _color(rng):
    return Color(*[int(v) / 255.0 for v in rng.randint(30, 256, size=3)], 1.0)


def _context(case, w, h):
    ctx = NewContext(w, h)
    ctx.Precision = PRECISION_MIXED if case["precision"] == "mixed" else PRECISION_PLAIN
    return ctx


def _clear(ctx):
    ctx.ClearColorBufferWith(scenes.BACKGROUND)
    ctx.ClearDepthBufferWith(FAR)


def prepare(case, seed):
    rng = _rng(case, seed)
    if case["kind"] == "frame":
        return _prepare_frame(case, rng)
    if case["kind"] in ("overlay", "lines"):
        s = case.get("scale", 1)
        w, h = case["width"] * s, case["height"] * s
        ctx = _context(case, w, h)
        eye = _eye(rng, 3.3)
        matrix = scenes.camera_matrix(w, h, eye=eye)
        return dict(case=case, ctx=ctx, mesh=_smoothed(_sphere_mesh(case, rng)), eye=eye,
                    shader=_phong(matrix, eye, _color(rng)),
                    overlay=NewSolidColorShader(matrix, (0, 0, 0, 0.5) if s > 1 else (0, 0, 0, 1)))
    if case["kind"] == "batch":
        return _prepare_batch(case, rng)
    p, n = _displaced(case["detail"], rng)
    t = p.shape[0]
    rec = np.zeros((t, 50), dtype=np.uint8)
    rec[:, 12:48] = p.float().cpu().numpy().reshape(t, 9).astype("<f4").view(np.uint8)
    return dict(case=case, stl=b"binary mesh".ljust(80, b" ") + struct.pack("<I", t) + rec.tobytes())


def _prepare_frame(case, rng):
    w, h = case["width"], case["height"]
    ctx = _context(case, w, h)
    if case["mesh"] == "lathe":
        mesh = _lathe_mesh(case["detail"], rng)
        eye = _eye(rng, 1.6)
        # near the surface, looking past the middle: some triangles cross the near plane and the frame's sides
        matrix = scenes.camera_matrix(w, h, eye=eye, center=V(0.2, 0.1, 0), fovy=60.0, near=0.5)
    else:
        mesh = _sphere_mesh(case, rng)
        eye = _eye(rng, 3.3)
        matrix = scenes.camera_matrix(w, h, eye=eye)
        if case["resident"]:
            mesh = _smoothed(mesh)
    if case["mesh"] == "lathe" and case["resident"]:
        mesh = DeviceMesh.upload(mesh)
    if case["shader"] == "texture":
        ctx.Shader = NewTextureShader(matrix, _texture(rng))
    else:
        ctx.Shader = _phong(matrix, eye, None if case["shader"] == "vertex" else _color(rng))
    return dict(case=case, ctx=ctx, mesh=mesh, matrix=matrix)


def _prepare_batch(case, rng):
    """views thumbnails, four to a mesh, of log-uniform meshes of 200 to 200,000 triangles at the
    benchmark's four resolutions. The sizes of the frames and meshes are the case's, their shapes
    and views the seed's."""
    batch, ctxs = Batch(), []
    s = case["scale"]
    plan = np.random.RandomState(case["views"])
    mesh = None
    for i in range(case["views"]):
        if i % 4 == 0:
            if plan.uniform() < 1.0 / 3:
                t = math.exp(plan.uniform(math.log(200), math.log(200000)))
                mesh = _smoothed(_sphere_mesh(dict(detail=int(min(6, max(2, round(math.log(t / 20.0, 4)))))), rng))
            else:
                mesh = DeviceMesh.upload(_lathe_mesh(int(math.exp(plan.uniform(math.log(8), math.log(512)))), rng))
        size = (256, 512, 768, 1024)[plan.randint(4)] * s
        eye = _eye(rng, 3.0)
        ctx = _context(case, size, size)
        ctx.Shader = _phong(scenes.camera_matrix(size, size, eye=eye, center=V(0, 0, 0)), eye, _color(rng))
        batch.Add(ctx, mesh, read_back=True, scale=s)
        ctxs.append(ctx)
    return dict(case=case, batch=batch, ctxs=ctxs)


# -- the calls ----------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "frame":
        ctx = state["ctx"]
        _clear(ctx)
        info = ctx.DrawMesh(state["mesh"])
        out = dict(image=ctx.Image(), info=list(info))
        if case["depth"]:
            out["depth"] = ctx.DepthBuffer
        return out
    if case["kind"] in ("overlay", "lines"):
        return _run_overlay(state)
    if case["kind"] == "batch":
        for ctx in state["ctxs"]:
            _clear(ctx)
        infos = state["batch"].Render()
        return dict(images=[state["batch"].Result(i) for i in range(len(infos))], infos=np.array(infos))
    mesh = DeviceMesh.load_stl(state["stl"])
    mesh.SmoothNormalsThreshold(Radians(case["degrees"]))
    mesh = mesh.download()
    return dict(positions=mesh.tri_pos, normals=mesh.tri_nrm)


def _run_overlay(state):
    case, ctx, mesh = state["case"], state["ctx"], state["mesh"]
    _clear(ctx)
    ctx.Shader = state["shader"]
    info = [ctx.DrawMesh(mesh)]
    ctx.Shader = state["overlay"]
    if case["kind"] == "overlay":
        ctx.Wireframe, ctx.DepthBias = True, 1e-5
        info.append(ctx.DrawMesh(mesh))
        image = ctx.Downsample(case["scale"])
    else:
        ctx.DepthBias = -1e-4
        info.append(ctx.DrawMesh(mesh.SharpEdges(Radians(40.0))))
        info.append(ctx.DrawMesh(mesh.Silhouette(state["eye"], 1e-3)))
        image = ctx.Image()
    ctx.Wireframe, ctx.DepthBias = False, 0.0
    return dict(image=image, infos=np.array(info))


# -- what a pass cannot do without ----------------------------------------------
def _draw_work(tris, pixels, per_vertex, shade):
    """Bytes and operations of one draw: every corner's attributes and index read once; about 50
    operations per distinct vertex, 46 for each of the front-facing half of the triangles, 12 for
    the coverage and depth and `shade` for the colour of each covered pixel (half the frame)."""
    return (tris * 3 * (per_vertex + 4), 25.0 * tris + 23.0 * tris + pixels * 0.5 * (12 + shade))


def work(case):
    if case["kind"] == "batch":
        px = case["views"] * 460000.0 * case["scale"] ** 2
        by, fl = _draw_work(case["views"] * 6000, px, 48, 121)
        return dict(bytes=by + case["views"] * 460000 * 4.0, flops=fl)
    t = 20 * 4 ** case["detail"] if case.get("mesh") != "lathe" else 4 * case["detail"]
    if case["kind"] == "prepare":
        return dict(bytes=50.0 * t + 2 * 72.0 * t, flops=120.0 * t)
    px = float(case["width"] * case["height"])
    s2 = case.get("scale", 1) ** 2
    per = 48 + {"texture": 16, "vertex": 32}.get(case.get("shader"), 0)
    by, fl = _draw_work(t, px * s2, per, 40 if case.get("shader") == "texture" else 121)
    by += 4 * px + (8 * px if case.get("depth") else 0)
    if case["kind"] == "overlay":
        fl += 3 * t * 2 * 46.0
    if case["kind"] == "lines":
        by += 2 * 3 * 24.0 * t
        fl += 120.0 * t
    return dict(bytes=by, flops=fl)


# -- 64-bit results, without the package ------------------------------------------
def exact(case, seed):
    if case["kind"] == "frame" and case["depth"]:
        return _exact_depth(case, seed)
    if case["kind"] == "prepare":
        return _exact_prepare(case, seed)
    return None


def _exact_depth(case, seed):
    """The depth buffer by plain torch: for each front-facing triangle the pixel centres inside
    it and the plane's depth there, the least of each pixel kept."""
    w, h = case["width"], case["height"]
    rng = _rng(case, seed)
    p, _ = _displaced(case["detail"], rng)
    m = torch.tensor(list(scenes.camera_matrix(w, h, eye=_eye(rng, 3.3))), dtype=torch.float64, device="cuda").reshape(4, 4)
    c = torch.cat([p, torch.ones_like(p[..., :1])], -1) @ m.T
    n = c[..., :3] / c[..., 3:]
    e = n[:, 1, :2] - n[:, 0, :2], n[:, 2, :2] - n[:, 0, :2]
    n = n[e[0][:, 0] * e[1][:, 1] - e[1][:, 0] * e[0][:, 1] > 0]
    x, y, z = (n[..., 0] + 1) * (w / 2), (1 - n[..., 1]) * (h / 2), (n[..., 2] + 1) / 2
    x0, x1 = x.amin(1).floor().clamp(0, w).long(), x.amax(1).ceil().clamp(0, w).long()
    y0, y1 = y.amin(1).floor().clamp(0, h).long(), y.amax(1).ceil().clamp(0, h).long()
    bw = (x1 - x0).clamp(min=0)
    count = bw * (y1 - y0).clamp(min=0)
    t = torch.repeat_interleave(torch.arange(count.numel(), device="cuda"), count)
    k = torch.arange(t.numel(), device="cuda") - (count.cumsum(0) - count)[t]
    px, py = x0[t] + k % bw[t], y0[t] + k // bw[t]
    b = []
    for i, j in ((1, 2), (2, 0), (0, 1)):
        b.append((x[t, j] - px - 0.5) * (y[t, i] - py - 0.5) - (y[t, j] - py - 0.5) * (x[t, i] - px - 0.5))
    area = b[0] + b[1] + b[2]
    b = [v / area for v in b]
    d = b[0] * z[t, 0] + b[1] * z[t, 1] + b[2] * z[t, 2]
    inside = (b[0] >= 0) & (b[1] >= 0) & (b[2] >= 0)
    depth = torch.full((h * w,), FAR, dtype=torch.float64, device="cuda")
    depth.scatter_reduce_(0, (py * w + px)[inside], d[inside], "amin")
    return dict(image=None, info=[None, None], depth=depth.reshape(h, w))


def _exact_prepare(case, seed):
    """Positions as the file has them; each corner's normal the normalised sum of the face normals
    at its position that are within the threshold of its own."""
    p, _ = _displaced(case["detail"], _rng(case, seed))
    p = p.float().double()
    n = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    n = (n / n.norm(dim=1, keepdim=True))[:, None, :].expand(-1, 3, -1).reshape(-1, 3)
    _, group, count = torch.unique(p.reshape(-1, 3), dim=0, return_inverse=True, return_counts=True)
    order = torch.argsort(group, stable=True)
    start = count.cumsum(0) - count
    total = torch.zeros_like(n)
    for k in range(int(count.max())):
        has = count[group] > k
        other = n[order[(start[group] + k).clamp(max=order.numel() - 1)]]
        take = has & ((other * n).sum(1) >= math.cos(math.radians(case["degrees"])))
        total += torch.where(take[:, None], other, torch.zeros_like(other))
    total /= total.norm(dim=1, keepdim=True)
    return dict(positions=p, normals=total.reshape(-1, 3, 3))
