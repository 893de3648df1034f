"""The work a program has this engine do, as measurable cases: whole frames (sync, lighting update, draw) of maps
from a few chunks to 64x32x64, draws alone, light baking, interactive edits, batched frames of many maps and
served requests.  Every case goes through the package's public calls (Volume, Image, Texture, Batch, Server) as a
host program makes them.  Maps are the seeded heightfields with boxes, spheres and lamps of
``doonengine_gb300.configs``; sizes are those of its configurations, of the tests and of ``bench.py``.

A case is a dict of plain values.  ``kind`` selects the program:

* ``frame``  one frame of a game loop: sync, lighting update, draw into an image in device memory
* ``host``   the same frame into an image in host memory, waited for (a program that shows or saves each frame)
* ``draw``   a moving camera over a lit map, no lighting update
* ``bake``   lighting updates of a still map, then the lighting read back (a light-map tool)
* ``edit``   a sphere placed into or cut out of the map, the edited chunks relit, a draw (an editor, a game's explosion)
* ``batch``  one batched frame of several maps (a renderer of many scenes)
* ``serve``  a draw, a relight and an edit per map through the request server, waited for
"""
import ctypes
import math
import random

import numpy as np
import torch

import doonengine_gb300 as dn
from doonengine_gb300.configs import build_volume

SKY_BOT, SKY_TOP = (0.30, 0.40, 0.55), (0.60, 0.80, 0.95)
EPS = 1e-4   # the reference's EPSILON (voxelShared.comp:7), part of its camera rays' definition


def _case(name, kind, map_size, res, K, **more):
    c = {"name": name, "kind": kind, "sx": map_size[0], "sy": map_size[1], "sz": map_size[2],
         "w": res[0], "h": res[1], "K": K,
         "shapes": 0,        # boxes and spheres strewn over the terrain
         "diffuse": 1,       # diffuse paths per voxel and update
         "spec_bounces": 2, "diff_bounces": 5,   # the reference's defaults
         "split": 1,         # lighting split of the sync: a chunk is relit every that many frames
         "rng": 0,           # 0: per-ray hash, 1: the reference's sine
         "glass": False,     # two of the materials transparent and refracting
         "raster": False,    # composed with a rasterised scene's colour and depth
         "view": 0,          # 0: lit; 1: albedo (the reference's view modes)
         "maps": 1}
    c.update(more)
    return c


def listed():
    return [
        # the smallest frame anybody draws: a preview or a thumbnail; launches and latency count
        _case("frame_tiny", "frame", (6, 5, 7), (96, 64), 8, shapes=6),
        # the small configuration of the benchmark: one room or prop at a low resolution
        _case("frame_small", "frame", (16, 16, 16), (640, 360), 16),
        # sizes that divide nothing, the library's default K, two paths per voxel, relit every third frame, the
        # reference's random numbers
        _case("frame_odd", "frame", (23, 11, 37), (317, 181), 15, shapes=90, diffuse=2, split=3, rng=1),
        # the headline workload: a whole landscape at full HD
        _case("frame_large", "frame", (64, 32, 64), (1920, 1080), 32, shapes=2000),
        # glass and water, composed with rasterised objects
        _case("frame_glass", "frame", (24, 12, 24), (960, 540), 16, shapes=120, glass=True, raster=True),
        # frames delivered to host memory
        _case("frame_host", "host", (24, 12, 24), (1280, 720), 16, shapes=120),
        # camera flights over the landscape, lighting at rest
        _case("draw_large", "draw", (64, 32, 64), (1920, 1080), 32, shapes=2000),
        # the unlit view an editor or a picker draws
        _case("draw_albedo", "draw", (12, 8, 12), (257, 143), 8, shapes=20, view=1),
        # light maps of a level: more paths and bounces than a game affords
        _case("bake", "bake", (16, 12, 16), (320, 180), 16, shapes=40, diffuse=4, spec_bounces=4),
        # edits while flying through a long map: only what was edited is relit
        _case("edit", "edit", (48, 16, 48), (1280, 720), 16, shapes=400, split=1 << 30),
        # a frame of many scenes at once
        _case("batch", "batch", (40, 32, 40), (1280, 720), 16, maps=12),
        # requests of many clients
        _case("serve", "serve", (24, 16, 24), (640, 360), 16, maps=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "host", "draw", "draw", "bake", "edit", "batch", "serve"])
    many = kind in ("batch", "serve")
    top = 32 if many else (20 if kind == "bake" else 64)
    size = (_log(rng, 5, top), _log(rng, 4, max(8, top // 2)), _log(rng, 5, top))
    w = _log(rng, 64, 1280 if many else 1920)
    h = max(36, min(1080, w * rng.choice([9, 9, 10, 12]) // 16 + rng.randrange(-3, 4)))
    c = _case("", kind, size, (w, h), rng.choice([4, 8, 13, 15, 16, 16, 24, 32]),
              shapes=rng.randrange(0, 1 + size[0] * size[2] // 4),
              diffuse=rng.choice([1, 1, 1, 2, 3]), split=rng.choice([1, 1, 2, 3]), rng=rng.choice([0, 0, 0, 1]),
              glass=rng.random() < 0.25, raster=kind in ("frame", "draw") and rng.random() < 0.25,
              view=rng.choice([0, 0, 1]) if kind == "draw" else 0)
    if kind == "bake":
        c.update(spec_bounces=rng.choice([1, 2, 3, 4]), diffuse=rng.choice([1, 2, 4]))
    if kind == "edit":
        c.update(split=1 << 30)
    if many:
        c.update(maps=rng.randrange(2, 13), raster=False)
    del c["name"]
    return c


# ---------------------------------------------------------------------- inputs

def _camera(rng, case):
    """A camera above the terrain looking across it, as the configurations place theirs."""
    return (rng.uniform(0.06, 0.14), 0.62 if case["sy"] < 32 else 0.42, rng.uniform(0.06, 0.14),
            rng.uniform(24.0, 34.0), rng.uniform(38.0, 50.0))


def _volume(case, rng, size=None, cpu_only=False):
    size = size or (case["sx"], case["sy"], case["sz"])
    tall = size[1] >= 32
    vol, _ = build_volume("small", cpu_only=cpu_only, map=size, seed=rng.randrange(1, 1 << 30),
                          mean=0.06 if tall else 0.26, amp=0.04 if tall else 0.14, shapes=case["shapes"],
                          shape_max=10 if tall else 18, K=case["K"], cam=_camera(rng, case))
    s = vol.s
    s.specBounceLimit, s.diffuseBounceLimit = case["spec_bounces"], case["diff_bounces"]
    s.rngMode, s.camViewMode = case["rng"], case["view"]
    for v, c in ((s.skyGradientBot, SKY_BOT), (s.skyGradientTop, SKY_TOP)):
        v.x, v.y, v.z = c
    if case["glass"]:
        vol.set_material(4, opacity=0.35, refract=1.33, specular=0.2, reflect_type=1, shininess=4)
        vol.set_material(9, opacity=0.6, refract=1.52, specular=0.3, reflect_type=1, shininess=6)
    return vol


class _View:
    """An image's memory as an array that keeps the image alive."""

    def __init__(self, image, field, typestr, shape):
        ptr = ctypes.cast(getattr(image.ptr.contents, field), ctypes.c_void_p).value
        self.image = image
        iface = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3, "strides": None}
        setattr(self, "__cuda_array_interface__" if image.on_device else "__array_interface__", iface)


def _outputs(image):
    views = {"color": _View(image, "color", "<f4", (image.height, image.width, 4)),
             "hit": _View(image, "hitIndex", "<i4", (image.height, image.width)),
             "face": _View(image, "hitFace", "|u1", (image.height, image.width))}
    if image.on_device:
        return {k: torch.as_tensor(v, device="cuda") for k, v in views.items()}
    return {k: np.asarray(v) for k, v in views.items()}


def _raster(case, nrng):
    """A rasterised scene: a few flat objects in front of an empty background (depth 1)."""
    w, h = max(16, case["w"] // 2), max(16, case["h"] // 2)
    color = nrng.random((h, w, 4), dtype=np.float32)
    depth = np.ones((h, w), np.float32)
    for _ in range(6):
        x, y = int(nrng.integers(0, w - 8)), int(nrng.integers(0, h - 8))
        depth[y:y + h // 6, x:x + w // 8] = nrng.uniform(0.975, 0.999)
    tex = dn.Texture(w, h, dn.Texture.RGBA32F), dn.Texture(w, h, dn.Texture.DEPTH32F)
    tex[0].upload(color)
    tex[1].upload(depth)
    return tex


def _views(vol, case, n=1, sweep=0.0):
    """View and projection matrices of n camera positions along a short flight."""
    aspect, out, yaw = case["w"] / case["h"], [], vol.s.camOrient.y
    for i in range(n):
        vol.s.camOrient.y = yaw + sweep * i
        out.append(vol.view_proj(aspect))
    vol.s.camOrient.y = yaw
    return out


def prepare(case, seed):
    dn.init()
    rng = random.Random(seed)
    nrng = np.random.default_rng(seed)
    st = {"case": case, "pass": 0}
    if case["maps"] > 1:
        return _prepare_many(case, rng, st)
    vol = _volume(case, rng)
    moving = case["kind"] == "draw"
    st.update(vol=vol, image=dn.Image(case["w"], case["h"], on_device=case["kind"] != "host"),
              views=_views(vol, case, 5 if moving else 1, 1.5 if moving else 0.0),
              raster=_raster(case, nrng) if case["raster"] else None)
    st["out"] = _outputs(st["image"])
    # the map streams in: chunks load one sync after a ray asked for them
    for i in range(10):
        view, proj = st["views"][i % len(st["views"])]
        vol.draw(st["image"], view, proj, st["raster"])
        vol.sync(dn.DN_READ_WRITE, 1)
        vol.update_lighting(case["diffuse"], 1000, 0.5 + i / 60.0)
    vol.finish()
    if case["kind"] == "bake":
        # the tool's own buffers: a row per lit voxel (at most 296 of a solid chunk's voxels are kept)
        n = 296 * vol.num_tiles * 2 // 3
        u32, f32 = ctypes.POINTER(ctypes.c_uint32), ctypes.POINTER(ctypes.c_float)
        st["rows"] = [(np.zeros(n, np.uint32), u32), (np.zeros((n, 3), np.float32), f32), (np.zeros((n, 3), np.float32), f32)]
    if case["kind"] == "edit":
        X, Y, Z = (8 * s for s in vol.map_size)
        r = max(3.0, min(11.0, 0.2 * min(X, Y, Z)))
        st["spots"] = [((rng.uniform(0.15, 0.5) * X, rng.uniform(0.22, 0.34) * Y, rng.uniform(0.15, 0.5) * Z),
                        rng.uniform(0.6, 1.0) * r, rng.randrange(0, 14), tuple(rng.randrange(40, 220) for _ in range(3)))
                       for _ in range(16)]
    return st


def _prepare_many(case, rng, st):
    vols, images, views = [], [], []
    for i in range(case["maps"]):
        # maps of many sizes, up to the case's, each with a resolution of its own
        f = [0.35 + 0.65 * ((i * g + 0.3) % 1.0) for g in (0.382, 0.618, 0.236, 0.472)]
        size = tuple(max(4, int(n * x)) for n, x in zip((case["sx"], case["sy"], case["sz"]), f))
        vols.append(_volume(case, rng, size))
        images.append(dn.Image(max(32, int(case["w"] * f[3])), max(32, int(case["h"] * f[3]))))
        views.append(vols[-1].view_proj(images[-1].width / images[-1].height))
    for i in range(10):
        for vol, image, vp in zip(vols, images, views):
            vol.draw(image, *vp)
            vol.sync(dn.DN_READ_WRITE, 1)
            vol.update_lighting(case["diffuse"], 1000, 0.5 + i / 60.0)
    for vol in vols:
        vol.finish()
    st.update(vols=vols, images=images, views=views, out=[_outputs(im) for im in images])
    if case["kind"] == "batch":
        st["batch"] = dn.Batch(vols)
        st["items"] = [dn.Batch.item(v, im, *vp, sync=(dn.DN_READ_WRITE, case["split"]), light=(case["diffuse"], 1000, 1.0))
                       for v, im, vp in zip(vols, images, views)]
    else:
        st["server"] = dn.Server(vols)
        st["server"].start()
        # an edit per map: a handful of voxels of its surface take a new material
        st["edits"] = [[((x, 1, z), (rng.randrange(8), 3, rng.randrange(8)), rng.randrange(14), (0.0, 1.0, 0.0),
                         (120, 140, 90), False) for x in range(1, 3) for z in range(1, 3)] for _ in vols]
    return st


# ---------------------------------------------------------------------- passes

def run(st):
    case, kind = st["case"], st["case"]["kind"]
    st["pass"] += 1
    t = 1.0 + st["pass"] / 60.0
    if kind == "batch":
        for it in st["items"]:
            it.time = t
        st["batch"].run(st["items"])
        return st["out"]
    if kind == "serve":
        return _serve(st, t)
    vol = st["vol"]
    view, proj = st["views"][st["pass"] % len(st["views"])]
    if kind == "draw":
        vol.draw(st["image"], view, proj, st["raster"])
        return st["out"]
    if kind == "bake":
        for i in range(4):
            vol.draw(st["image"], view, proj)
            vol.sync(dn.DN_READ_WRITE, 1)
            vol.update_lighting(case["diffuse"], 1000, t + i / 240.0)
        rows = st["rows"]
        n = vol.lib.DN_export_lighting(vol.ptr, *(a.ctypes.data_as(p) for a, p in rows), len(rows[0][0]))
        if n > len(rows[0][0]):
            raise RuntimeError("more lit voxels than rows")
        return {"index": rows[0][0].view(np.int32), "diffuse": rows[1][0], "specular": rows[2][0]}
    if kind == "edit":
        n = st["pass"] - 1
        center, radius, material, albedo = st["spots"][n % len(st["spots"])]
        vol.shape("sphere", (255 if n % 2 else material, (0.0, 1.0, 0.0), albedo), center, a=radius, flip=bool(n % 2))
    vol.sync(dn.DN_READ_WRITE, case["split"])
    vol.update_lighting(case["diffuse"], 1000, t)
    vol.draw(st["image"], view, proj, st["raster"])
    if kind == "host":
        vol.finish()
    return st["out"]


def _serve(st, t):
    srv = st["server"]
    for i, (image, vp) in enumerate(zip(st["images"], st["views"])):
        srv.submit(srv.relight_request(i, st["case"]["diffuse"], 1000, t))
        srv.submit(srv.edit_request(i, st["edits"][i]))
        srv.submit(srv.draw_request(i, image, *vp))
    srv.drain(60.0)
    srv._keep.clear()   # the edits of finished requests
    if not all(c["ok"] for c in srv.poll()):
        raise RuntimeError("a request failed")
    return st["out"]


# ---------------------------------------------------------------------- what a pass cannot do without

def work(case):
    """Each array once: the per-tile state, the occupancy masks, voxel words and lighting of the chunks in view,
    the new lighting, the image.  Operations: a dozen per cell a ray visits, some twenty cells per ray."""
    tiles = case["sx"] * case["sy"] * case["sz"]
    pixels = case["w"] * case["h"]
    scenes = case["maps"] * (0.3 if case["maps"] > 1 else 1.0)   # sizes and resolutions drawn up to the case's
    columns = case["sx"] * case["sz"]
    chunks = 1.5 * columns            # surface chunks in view
    voxels = 200 * chunks             # kept voxels of a surface chunk (its underground faces among them)
    kind = case["kind"]
    lit = 0.0 if kind == "draw" else voxels / min(case["split"], 30)
    updates = 4 if kind == "bake" else 1
    bytes_ = chunks * 128 + voxels * 40 + updates * (tiles * 8 + lit * 40) + pixels * 21
    if kind == "bake":
        bytes_ += voxels * 28
    rays = updates * (lit * (2.2 * case["K"] + 2.5 * case["diffuse"])) + pixels * (4 if kind == "bake" else 1)
    return {"bytes": scenes * bytes_, "flops": scenes * rays * 20 * 12}


# ---------------------------------------------------------------------- 64-bit results

def exact(case, seed):
    """The unlit draw in 64 bits: every pixel's ray walked through the dense voxel grid.  The hit index and face
    are whole numbers, compared as such.  Lit results have no such value: which voxel a ray of the lighting update
    reaches is decided by the 32-bit steps the engine defines (and by its random numbers), and a 64-bit walk
    reaches others; nor has a refracting or composed draw.  None also for maps that take long in numpy."""
    if case["kind"] != "draw" or case["view"] != 1 or case["glass"] or case["raster"] or case["w"] * case["h"] > 150000:
        return None
    if case["sx"] * case["sy"] * case["sz"] > 12000:
        return None
    vol = _volume(case, random.Random(seed), cpu_only=True)
    X, Y, Z = (8 * s for s in vol.map_size)
    normal, albedo, _ = vol.export_voxels()
    solid = ((normal >> 24) != 255) & (normal != 0xFFFFFFFF)
    view, proj = (dn.volume.mat_to_np(m).astype(np.float64).T for m in _views(vol, case, 5, 1.5)[1])
    pos = np.linalg.inv(view)[:3, 3]
    centered = view.copy()
    centered[:3, 3] = 0.0
    M = np.linalg.inv(centered) @ np.linalg.inv(proj)
    w, h = case["w"], case["h"]
    px, py = np.meshgrid(np.arange(w) / w * 2 - 1, np.arange(h) / h * 2 - 1)
    d = (M @ np.stack([px.ravel(), py.ravel(), np.zeros(w * h), np.ones(w * h)]))[:3].T
    d = d / np.linalg.norm(d, axis=1, keepdims=True) + EPS
    # distances in chunks; the grid in voxels
    lo, hi = (0 - pos) / d, (np.array([X, Y, Z]) / 8 - pos) / d
    near, far = np.minimum(lo, hi).max(1), np.maximum(lo, hi).min(1)
    inside = (near <= far) & (far >= 0)
    start = np.where(near > 0, near + EPS, 0.0)
    p = (pos + d * start[:, None]) * 8
    cell = np.floor(p).astype(np.int64)
    step = np.sign(d).astype(np.int64)
    delta = 1 / np.abs(d)
    side = np.where(d > 0, cell + 1 - p, p - cell) * delta
    size = np.array([X, Y, Z])
    table = np.array([int(math.pow(b / 255, 2.2) * 255) for b in range(256)]) / 255.0
    a = (d[:, 1:2] * 0.5 + 1.0)
    sky = np.array(SKY_BOT) * (1 - a) + np.array(SKY_TOP) * a
    out = np.concatenate([sky ** (2.2 * 0.4545), np.full((w * h, 1), -1.0)], 1)
    live = np.flatnonzero(inside)
    last = np.zeros(w * h)
    while live.size:
        c = cell[live]
        ok = ((c >= 0) & (c < size)).all(1)
        live, c = live[ok], c[ok]
        at = c[:, 0] + X * (c[:, 1] + Y * c[:, 2])
        hit = solid[at]
        i, word = live[hit], albedo[at[hit]]
        rgb = np.stack([table[(word >> k) & 255] for k in (24, 16, 8)], 1)
        out[i, :3] = rgb ** 0.4545
        out[i, 3] = np.linalg.norm(d[i], axis=1) * (start[i] + last[i] / 8 + EPS / 8)
        live = live[~hit]
        s = side[live]
        last[live] = s.min(1)
        m = s == s.min(1, keepdims=True)
        side[live] = s + m * delta[live]
        cell[live] += m * step[live]
    vol.close()
    return {"color": out.reshape(h, w, 4), "hit": None, "face": None}
