"""The work that a program using this renderer has it do, as measurable cases.

A case is one step of a real program: a frame with its shadow cascades, a
view of a scene whose shadow maps stand, a pose change with its vertex
light, the post effects, a displayed frame, a batch of views read back.  The
scenes are seeded terrain, icospheres and alpha-tested quads of the shapes
in axi_visualizer_b200/scenes.py.

Kinds and their ranges (draw() spreads over them; widths are multiples of 16
as the framebuffer wants them, heights any number):
  frame    2,500 to 2,900,000 triangles, 320x180 to 3840x2160, one or two
           cascades of 256 to 4096 a side; trilinear or plain textures,
           alpha-tested quads and alpha-tested terrain bands
  normal   the normal-mapped materials, shadow maps standing
  multi    the 4-way blend terrain, shadow maps standing
  pose     rotate / translate / vertLight of a group, its vertices read back
  anim     a frame in which the sphere groups turn and all light is redone
  post     ssao, dof, blur and gamma on a frame already on the device
  display  ssao and blur, then the 8-bit frame in host memory
  batch    cascades, a main view and six cube faces in one batch, the shaded
           views read back to pinned memory
"""
import math

import numpy as np
import torch

from axi_visualizer_b200 import scenes as S
from axi_visualizer_b200.batch import PHASED, Batch, cube_faces, depth, shaded
from axi_visualizer_b200.ops import SKY_COLOR, CLDraw

AMB = 0.2
BIAS = 0.2


def _frame(name, w, h, terrain_n, spheres, quads, extent, spread, tex, alpha_tex, casc0, casc1, mip=1, bands=1,
           alpha_bands=0):
    return dict(name=name, kind="frame", w=w, h=h, terrain_n=terrain_n, spheres=spheres, quads=quads, extent=extent,
                spread=spread, tex=tex, alpha_tex=alpha_tex, casc0=casc0, casc1=casc1, mip=mip, bands=bands,
                alpha_bands=alpha_bands)


def listed():
    return [
        # an editor's preview pane or a thumbnail: launches and latency, the smallest frame of the parity tests
        _frame("frame_tiny", 320, 192, 16, 24, 40, 16.0, 12.0, 64, 64, 256, 128),
        # the plain 640x480 view of 24,192 triangles with one cascade
        _frame("frame_vga", 640, 480, 64, 200, 0, 32.0, 20.0, 512, 512, 1024, 0),
        # a served scene of ordinary size at 720p; spheres without mips, a few alpha quads
        _frame("frame_720p_300k", 1280, 720, 274, 1690, 7500, 42.0, 25.0, 1024, 512, 2048, 1024, mip=0),
        # the benchmark's frame: 1080p, 1,044,288 triangles, two 2048 cascades
        _frame("frame_1080p_1m", 1920, 1080, 512, 6000, 20000, 64.0, 20.0, 2048, 1024, 2048, 2048, bands=2),
        # the 4K stress view, about a third of it alpha-tested terrain, 4096 cascades
        _frame("frame_4k_2900k", 3840, 2160, 1024, 10000, 0, 96.0, 36.0, 2048, 2048, 4096, 4096, bands=4, alpha_bands=1),
        # the normal-mapped materials at an odd height (a window, not a screen mode)
        dict(name="normal_1296x713", kind="normal", w=1296, h=713, terrain_n=128, spheres=400, quads=1000, extent=32.0,
             spread=20.0, tex=512, casc0=2048),
        # a heightfield landscape in the 4-way blend material, as the terrain demo draws it
        dict(name="multi_1080p", kind="multi", w=1920, h=1080, terrain_n=192, cell=1.0, spheres=64, tex=512, casc0=2048),
        # one object posed and its vertices read back (collision, picking): a handful of short calls
        dict(name="pose_1280", kind="pose", tris=1280, dirs=3, points=2, spots=1),
        # an animated scene: the sphere groups turn, every vertex is lit by 3 + 8 + 4 lights, then the view
        dict(name="anim_720p_500k", kind="anim", w=1280, h=720, terrain_n=360, spheres=3000, quads=2000, extent=48.0,
             spread=20.0, tex=1024, alpha_tex=512, casc0=1024, dirs=3, points=8, spots=4),
        # all post effects of a 1080p frame
        dict(name="post_1080p", kind="post", w=1920, h=1080, focus=12.0),
        # a small window at an odd height, shown: effects, then 8-bit RGB in pinned host memory
        dict(name="display_848x477", kind="display", w=848, h=477, exposure=1.0),
        # reflections: two cascades, the main view and a cube map around the eye in one batch
        dict(name="batch_cube", kind="batch", w=1280, h=720, face=256, terrain_n=64, spheres=200, extent=32.0,
             spread=20.0, tex=512, casc0=2048, casc1=1024),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, lo, hi):
    w = max(1, round(_log(rng, lo, hi) / 16)) * 16
    return w, max(32, int(w * rng.uniform(0.5, 0.75)))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["normal", "multi", "pose", "anim", "post", "display", "batch"])
    side = lambda lo, hi: 2 ** rng.randint(lo, hi)   # noqa: E731
    if kind == "frame":
        t = _log(rng, 2500, 2000000)
        w, h = _size(rng, 320, 2560)
        tex = side(6, 10)
        bands = rng.randint(1, 4)
        quads = int(t * rng.uniform(0.0, 0.1) / 2)
        ab = rng.choice([0, 0, 1]) if bands > 1 else 0
        c = _frame("", w, h, max(8, round(math.sqrt(t * 0.25))), max(2, int(t * rng.uniform(0.3, 0.45) / 80)), quads,
                   round(rng.uniform(16, 64), 2), round(rng.uniform(10, 30), 2), tex, tex if ab else side(6, 9),
                   side(8, 11) + rng.choice([0, 0, 40]), rng.choice([0, side(8, 11)]), rng.randint(0, 1), bands, ab)
        del c["name"]
        return c
    if kind == "normal":
        w, h = _size(rng, 320, 1920)
        return dict(kind=kind, w=w, h=h, terrain_n=rng.randint(16, 160), spheres=rng.randint(20, 500),
                    quads=rng.randint(30, 1500), extent=32.0, spread=20.0, tex=side(6, 9), casc0=side(8, 11))
    if kind == "multi":
        w, h = _size(rng, 320, 1920)
        return dict(kind=kind, w=w, h=h, terrain_n=rng.randint(24, 256), cell=round(rng.uniform(0.5, 2), 2),
                    spheres=rng.randint(12, 100), tex=side(6, 9), casc0=side(8, 11))
    if kind == "pose":
        return dict(kind=kind, tris=int(_log(rng, 80, 20000)), dirs=rng.randint(1, 3), points=rng.randint(0, 5),
                    spots=rng.randint(0, 3))
    if kind == "anim":
        w, h = _size(rng, 320, 1280)
        return dict(kind=kind, w=w, h=h, terrain_n=rng.randint(32, 360), spheres=int(_log(rng, 100, 3000)),
                    quads=rng.randint(0, 2000), extent=48.0, spread=20.0, tex=side(6, 10), alpha_tex=side(6, 9),
                    casc0=side(8, 11), dirs=rng.randint(1, 3), points=rng.randint(0, 16), spots=rng.randint(0, 8))
    if kind in ("post", "display"):
        w, h = _size(rng, 256, 2560)
        c = dict(kind=kind, w=w, h=h)
        c.update(dict(focus=round(rng.uniform(2, 40), 2)) if kind == "post" else dict(exposure=round(rng.uniform(0.5, 2), 2)))
        return c
    w, h = _size(rng, 320, 1280)
    return dict(kind=kind, w=w, h=h, face=16 * rng.randint(4, 24), terrain_n=rng.randint(16, 128),
                spheres=rng.randint(20, 600), extent=32.0, spread=20.0, tex=side(6, 9), casc0=side(8, 11),
                casc1=side(8, 11))


# ---------------------------------------------------------------- scenes

def _texture(rng, n, mip):
    return S.texture_planes(S.noise_rgb_fast(rng, n), bool(mip))[0]


class Scene:
    """A CLDraw with its groups, materials and cameras, as an engine keeps it."""

    def __init__(self, w, h, pinned=False):
        self.draw = CLDraw(1, 64, w, h, 1, pinned=pinned)
        self.draw.setPrimaryLight(np.asarray(S.LIGHT_INTS[:1]), np.asarray(S.LIGHT_DIRS[:1]))
        self.view = S.default_view(w, h)
        self.shaders, self.cast, self.shadows = [], [], []

    def add(self, mesh, planes, shader, mip=0):
        xyz, vn, uv = mesh
        tn = self.draw.addTextureGroup(xyz, uv, vn, *planes, mip=mip or False)
        self.shaders.append(shader)
        self.cast.append(True)
        return tn

    def light(self, dirs=3):
        mask = np.ones(len(self.shaders), np.uint8)
        self.draw.ambLight = np.float32(AMB)
        self.draw.vertLight(mask, np.asarray(S.LIGHT_INTS[:dirs]), np.asarray(S.LIGHT_DIRS[:dirs]))

    def cascade(self, dim, half_extent):
        if not dim:
            return
        k = len(self.shadows)
        cam = S.ShadowCam.facing(dim, dim / 2 / half_extent, (0, 0, 0), S.SUN)
        self.draw.addShadowMap(k, cam.dim, cam.scale, AMB)
        self.draw.placeShadowMapBasis(k, cam.pos, cam.vv, AMB)
        self.shadows.append(cam)

    def shadow_pass(self):
        for k in range(len(self.shadows)):
            self.draw.clearShadowMap(k)
            self.draw.shadowMap(k, self.cast, self.shaders, BIAS)

    def main_view(self):
        d, v = self.draw, self.view
        d.setScaleCull(v.sscale, v.cax, v.cay)
        d.setPos(v.pos)
        d.setVM(v.vv)
        d.clearZBuffer()
        d.clearColor(SKY_COLOR)
        d.drawAll(self.shaders, shadowIds=list(range(len(self.shadows))))


def _split(mesh, parts):
    n = len(mesh[0]) // 3
    cut = [3 * (n * k // parts) for k in range(parts + 1)]
    return [tuple(a[cut[k]:cut[k + 1]] for a in mesh) for k in range(parts)]


def _f32(mesh):
    return tuple(np.ascontiguousarray(a, np.float32) for a in mesh)


def _mixed(case, seed, pinned=False):
    """Terrain in `bands` groups (the last `alpha_bands` of them alpha-tested),
    two groups of spheres, alpha-tested quads."""
    rng = np.random.default_rng(seed)
    sc = Scene(case["w"], case["h"], pinned)
    n, e, sp = case["terrain_n"], case["extent"], case["spread"]
    tex, mip = case["tex"], case.get("mip", 1)
    flags = "mip shadow" if mip else "shadow"
    chain = tex if mip else 0
    ground, skin = _texture(rng, tex, mip), _texture(rng, tex, mip)
    cell = 2 * e / n
    bands = case.get("bands", 1)
    if case.get("quads") or case.get("alpha_bands"):
        a = case["alpha_tex"]
        sc.draw.addTexAlpha(rng.random((a, a)) < 0.6)
    for k, part in enumerate(_split(_f32(S.terrain(rng, n, cell, (-e, 0.0, -e), min(2.0, 2.0 * cell))), bands)):
        alpha = k >= bands - case.get("alpha_bands", 0)
        sc.add(part, ground, dict({f: 1 for f in flags.split()}, alpha=0) if alpha else flags, chain)
    for part in _split(_f32(S.icospheres(rng, case["spheres"], 0.2, 1.0, -sp, sp)), 2):
        sc.add(part, skin, flags + " cull", chain)
    if case.get("quads"):
        sc.add(_f32(S.quads(rng, case["quads"], -sp, sp, 0.3, 1.0)), _texture(rng, case["alpha_tex"], 0),
               {"alpha": 0, "shadow": 1})
    sc.light()
    sc.cascade(case.get("casc0", 0), 1.2 * sp)
    sc.cascade(case.get("casc1", 0), 1.15 * e)
    return sc


def _normal_scene(case, seed):
    rng = np.random.default_rng(seed)
    sc = Scene(case["w"], case["h"])
    n, e, sp, tex = case["terrain_n"], case["extent"], case["spread"], case["tex"]
    for name, mip in (("flat", False), ("chain", True)):
        sc.draw.addNrmMap(S.normal_map(rng, tex, mip), name)
    sc.draw.addTexAlpha(rng.random((tex, tex)) < 0.6)
    plain, chain = _texture(rng, tex, 0), _texture(rng, tex, 1)
    s1, s2 = _split(_f32(S.icospheres(rng, case["spheres"], 0.5, 2.0, -sp, sp)), 2)
    sc.add(_f32(S.terrain(rng, n, 2 * e / n, (-e, 0.0, -e), 1.0, 2.0)), plain, {"normal": ("flat", 0.5), "shadow": 1})
    sc.add(s1, plain, {"normal": ("flat", 0.3), "metal": 1, "shadow": 1, "cull": 1})
    sc.add(s2, chain, {"normal": ("chain", 0.5), "mip": np.float32(0.4), "shadow": 1, "cull": 1}, tex)
    sc.add(_f32(S.quads(rng, case["quads"], -sp, sp, 0.5, 2.0)), plain, {"normal": ("flat", 0.7), "alpha": 0, "shadow": 1})
    sc.light()
    sc.cascade(case["casc0"], 1.2 * sp)
    return sc


def _multi_scene(case, seed):
    rng = np.random.default_rng(seed)
    sc = Scene(case["w"], case["h"])
    n, cell, tex = case["terrain_n"], case["cell"], case["tex"]
    i = np.arange(n + 1) * cell
    hx, hz = np.meshgrid(i, i, indexing="ij")
    h = 12.5 + 9.0 * np.sin(hx * 0.225 + rng.uniform(0, 6)) * np.cos(hz * 0.175 + rng.uniform(0, 6))
    h += rng.standard_normal(h.shape) * 0.5
    e = n * cell / 2
    sc.add(_f32(S.terrain_from_heights(h, cell, (-e, 0.0, -e), 8.0 * cell)), _texture(rng, tex, 0), "multi cull")
    for k in range(3):
        sc.add(_f32(S.quads(rng, 1, -4, 4, 1.0, 2.0, ground=26.0)), _texture(rng, tex, 0), "")
    sx, sn, su = S.icospheres(rng, case["spheres"], 0.5, 2.0, -e / 2, e / 2)
    sx[:, 1] = sx[:, 1] * 0.2 + 22.0
    sc.add(_f32((sx, sn, su)), _texture(rng, tex, 1), "mip shadow cull", tex)
    sc.view = S.default_view(case["w"], case["h"], pos=(0.0, 30.0, -0.9 * e), target=(0.0, 10.0, 0.0))
    sc.light()
    sc.cascade(case["casc0"], 1.2 * e)
    return sc


def _lights(rng, case, spread):
    pts = rng.uniform(-spread, spread, (case["points"], 3)), rng.uniform(0.5, 4.0, (case["points"], 3))
    d = rng.standard_normal((case["spots"], 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    spots = rng.uniform(-spread, spread, (case["spots"], 3)), d, rng.uniform(0.5, 4.0, (case["spots"], 3))
    f = lambda a: np.ascontiguousarray(a, np.float32)   # noqa: E731
    return dict(dirI=f(S.LIGHT_INTS[:case["dirs"]]), dirD=f(S.LIGHT_DIRS[:case["dirs"]]), pointI=f(pts[1]),
                pointP=f(pts[0]), spotI=f(spots[2]), spotD=f(spots[1]), spotP=f(spots[0]))


def _turn(a):
    c, s = math.cos(a), math.sin(a)
    return np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]], np.float32)


def _pose_inputs(case, seed):
    """The object's mesh and what moves and lights it, plain numpy."""
    rng = np.random.default_rng(seed)
    mesh = _f32(S.icospheres(rng, -(-case["tris"] // 80), 0.2, 1.0, -4, 4))
    mesh = tuple(a[:3 * case["tris"]] for a in mesh)
    return dict(mesh=mesh, old=_turn(-0.3), rot=_turn(0.35), origin=np.array([0.5, -0.25, 1.0], np.float32),
                shift=rng.uniform(-0.5, 0.5, 3).astype(np.float32), first=int(rng.integers(1, 3 * case["tris"] // 2)),
                lights=_lights(rng, case, 6.0), planes=_texture(rng, 64, 0))


class _Device:
    """A device buffer of a handle, as an array torch can view; it keeps the
    handle, whose end frees the buffer."""

    def __init__(self, draw, ptr, shape, typestr):
        self.draw = draw
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _planes(draw):
    """The handle's frame on the device: three 16-bit colour planes and the depth."""
    r, g, b, z, _ = draw.device_ptrs()
    shape = (draw.H, draw.W)
    return [torch.as_tensor(_Device(draw, p, shape, t), device="cuda")
            for p, t in ((r, "<i2"), (g, "<i2"), (b, "<i2"), (z, "<f4"))]


# ---------------------------------------------------------------- the cases

def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        sc = _mixed(case, seed)
        return dict(kind=kind, sc=sc, out=_planes(sc.draw))
    if kind in ("normal", "multi"):
        sc = _normal_scene(case, seed) if kind == "normal" else _multi_scene(case, seed)
        sc.shadow_pass()
        return dict(kind=kind, sc=sc, out=_planes(sc.draw))
    if kind == "pose":
        p = _pose_inputs(case, seed)
        sc = Scene(64, 64)
        sc.add(p["mesh"], p["planes"], "")
        sc.draw.ambLight = np.float32(AMB)
        return dict(kind=kind, sc=sc, p=p)
    if kind == "anim":
        sc = _mixed(case, seed)
        sc.shadow_pass()
        return dict(kind=kind, sc=sc, lights=_lights(np.random.default_rng(seed + 1), case, 20.0), old=_turn(0.0),
                    rot=_turn(0.01), mask=np.ones(len(sc.shaders), np.uint8), out=_planes(sc.draw))
    if kind in ("post", "display"):
        # a frame that something else on the device hands over: depth in place, colour copied in each time
        sc = _mixed(dict(w=case["w"], h=case["h"], terrain_n=64, spheres=200, extent=32.0, spread=20.0, tex=256,
                         casc0=1024), seed, pinned=True)
        sc.shadow_pass()
        sc.main_view()
        sc.draw.sync()
        planes = _planes(sc.draw)
        return dict(kind=kind, sc=sc, case=dict(case), out=planes[:3], given=[p.clone() for p in planes[:3]],
                    rand=np.random.default_rng(seed).random(48).astype(np.float32), waiting=None,
                    stream=torch.cuda.ExternalStream(sc.draw.stream_ptr()))
    if kind == "batch":
        sc = _mixed(case, seed)
        eye = (0.0, 5.0, -25.0)
        views = [depth(c, BIAS) for c in sc.shadows]
        nd = len(views)
        views += [shaded(v, list(range(nd)), clear=SKY_COLOR) for v in [sc.view] + cube_faces(eye, case["face"])]
        b = Batch(sc.draw, views)
        b.set_mode(PHASED)
        host = []
        for d in views[nd:]:
            host.append([torch.empty((d.h, d.w), dtype=t, pin_memory=True) for t in (torch.int16,) * 3 + (torch.float32,)])
        return dict(kind=kind, sc=sc, batch=b, nd=nd, out=host, into=[[p.numpy() for p in v] for v in host],
                    flags=[S.flags_from_string(s) for s in sc.shaders])
    raise ValueError(kind)


def run(state):
    kind, sc = state["kind"], state["sc"]
    d = sc.draw
    if kind == "frame":
        sc.shadow_pass()
        sc.main_view()
        return state["out"]
    if kind in ("normal", "multi"):
        sc.main_view()
        return state["out"]
    if kind == "pose":
        p = state["p"]
        d.rotate(p["old"], p["rot"], p["origin"], 0, None, 0)
        d.translate(p["shift"], p["first"], None, 0)
        d.vertLight([1], **p["lights"])
        return d.getVertices(0)
    if kind == "anim":
        spheres = [k for k, s in enumerate(sc.shaders) if "cull" in s]
        for tn in spheres:
            d.rotate(state["old"], state["rot"], (0.0, 0.0, 0.0), 0, None, tn)
        d.vertLight(state["mask"], **state["lights"])
        sc.main_view()
        return state["out"]
    if kind in ("post", "display"):
        with torch.cuda.stream(state["stream"]):
            for to, given in zip(state["out"], state["given"]):
                to.copy_(given)
        d.ssao(state["rand"])
        if kind == "post":
            d.dof(state["case"]["focus"])
            d.blur()
            d.gamma(1.0)
            return state["out"]
        d.blur()
        # the next frame is issued before the last one is awaited
        ticket = d.readFrameRGB8Async(state["case"]["exposure"])
        if state["waiting"] is not None:
            d.waitFrame(state["waiting"])
        state["waiting"] = ticket
        return ticket[1]
    if kind == "batch":
        b = state["batch"]
        b.render(state["flags"])
        for k, planes in enumerate(state["into"]):
            b.read_async(state["nd"] + k, *planes)
        return state["out"]
    raise ValueError(kind)


def _tris(case):
    return (2 * case["terrain_n"] ** 2 + 80 * case["spheres"] + 2 * case.get("quads", 0), 2 * case.get("quads", 0) +
            2 * case["terrain_n"] ** 2 * case.get("alpha_bands", 0) // case.get("bands", 1))


def work(case):
    """Bytes of one pass, inputs and outputs once each: 132 a triangle of a
    view (positions, normals, light, uv), 36 a caster (60 alpha-tested) and 4 a
    texel of each cascade, 10 a pixel; 72 a turned vertex-triangle's data and so
    on for the vertex stage.  Operations: those of a triangle's projection."""
    kind = case["kind"]
    if kind == "pose":
        t = case["tris"]
        n = 3 * t
        return {"bytes": n * 60.0, "flops": n * (60.0 + 10 * case["dirs"] + 25 * case["points"] + 35 * case["spots"])}
    px = case["w"] * case["h"]
    if kind in ("post", "display"):
        return {"bytes": px * (16.0 if kind == "post" else 13.0), "flops": px * 16 * 25.0}
    t, alpha = _tris(case)
    b, f = 132.0 * t + 10.0 * px, 60.0 * t + 100.0 * px
    if kind in ("frame", "batch"):
        for dim in (case["casc0"], case["casc1"]):
            if dim:
                b += 36.0 * t + 24.0 * alpha + 4.0 * dim * dim
                f += 50.0 * t
    if kind == "batch":
        b += 6 * 10.0 * case["face"] ** 2 + 6 * 36.0 * t
        f += 6 * 60.0 * t
    if kind == "anim":
        n = 3 * t
        b += n * 36.0 + 80 * 3 * case["spheres"] * 48.0
        f += n * (10.0 * case["dirs"] + 25 * case["points"] + 35 * case["spots"])
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """The posed vertices in 64 bits.  The other kinds give 16-bit colour and
    the depth of whichever fragment 32-bit scan conversion lets win, which has
    no 64-bit counterpart."""
    if case["kind"] != "pose":
        return None
    p = _pose_inputs(case, seed)
    xyz, vn, _ = (np.asarray(a, np.float64) for a in p["mesh"])
    old, rot, o = (np.asarray(p[k], np.float64) for k in ("old", "rot", "origin"))
    xyz = (xyz - o) @ old.T @ rot + o
    vn = vn @ old.T @ rot
    xyz[p["first"]:] += np.asarray(p["shift"], np.float64)
    L = {k: np.asarray(v, np.float64) for k, v in p["lights"].items()}
    li = np.zeros_like(vn)
    for d, i in zip(L["dirD"][1:], L["dirI"][1:]):
        li += (np.maximum(0.0, vn @ d + 0.5) * np.float64(np.float32(0.66)))[:, None] * i
    for q, i in zip(L["pointP"], L["pointI"]):
        v = xyz - q
        r = np.linalg.norm(v, axis=1)
        nd = np.einsum("ij,ij->i", vn, v)
        li += (np.where(nd > 0, nd / r / (1 + r * r), 0.0))[:, None] * i
    for q, d, i in zip(L["spotP"], L["spotD"], L["spotI"]):
        v = xyz - q
        r = np.linalg.norm(v, axis=1)
        nd, sd = np.einsum("ij,ij->i", vn, v), v @ d
        li += (np.where((nd > 0) & (sd > 0), nd / r * (sd / r) / (1.5 + r * r), 0.0))[:, None] * i
    return xyz, vn, np.maximum(li, np.float64(np.float32(AMB)))
