"""The work that a user of the render core has it do, as cases that can be timed.

Each case is one pass through the public entry points (include/crg.h, or the
thin handles over it in crender_gb300/api.py) on inputs resident on the GPU,
with the scene built and the buffers allocated beforehand, as an application
keeps them.  Workloads and sizes are the ones of scenes.py and the benchmark:
the box scene, the displaced sphere (up to 4,195,280 triangles) on a ground
quad under a sphere light, the random triangle soup, the box as three models
with instances, the inverse-rendering box, and a 3840x2160 image.

  pick      closest hits of a few rays on a mesh: mouse picking, autofocus
  closest   closest hits of millions of incoherent rays (the traversal benchmark)
  any       occlusion of millions of incoherent shadow rays
  render    crg_render, the drop-in for a renderer's sample passes: box or mesh,
            both estimators, FP32 film with or without the FP64 planes
  viewport  one interactive refresh: reset, a few samples with the reference
            estimator (sun, image sky, instances), display transform
  batch     crg_render_batch: many views of uneven size and spp in one launch
  inverse   one step of inverse rendering: forward, L2 loss, adjoint
  post      the post-processing chain on a finished image
  rebuild   a resident mesh rebuilt under two sets of build options and queried,
            as a search for the best BVH does
  dynamic   the build without allocation of a mesh that changes every frame
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from crender_gb300 import _abi, api, scenes

_CTX = []


def context():
    """The process's one render context."""
    if not _CTX:
        _CTX.append(api.Context(0))
    return _CTX[0]


class _Held:
    """Closes a handle when the last thing that uses it goes."""

    def __init__(self, x):
        self.x = x

    def __del__(self):
        (self.x.close if hasattr(self.x, "close") else self.x.free)()


class _Memory:
    """Device memory of a library handle, which lives at least as long as the views of it."""

    def __init__(self, held, ptr, shape, typestr):
        self.held = held
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, data=(int(ptr), False), version=3,
                                             strides=None)


def _tensor(held, ptr, shape, dtype):
    """A torch view of `shape` over device memory that `held`'s handle owns."""
    t = torch.as_tensor(_Memory(held, ptr, shape, "<f4" if dtype == torch.float32 else "<f8"), device="cuda")
    t.held = held
    return t


class State:
    """What a program holds between calls; a handle is closed when neither it nor an output uses it."""

    def __init__(self, kind):
        self.kind = kind
        self.held = []

    def own(self, x):
        self.held.append(_Held(x))
        return x


# ----------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


_GRID = {}


def _grid(freq):
    """Points and triangles of the geodesic grid (scenes.geodesic_grid), on the GPU."""
    if freq not in _GRID:
        if len(_GRID) >= 4:
            _GRID.clear()
        pts, local = scenes.geodesic_grid(freq)
        _GRID[freq] = (torch.from_numpy(pts).cuda(), torch.from_numpy(local).cuda())
    return _GRID[freq]


def _sphere(freq, g):
    """Triangles float32 [20 * freq^2, 9] of the unit geodesic sphere displaced radially by six
    octaves of waves (gain 1/2, lacunarity 2, amplitude 0.05), wound outwards."""
    pts, local = _grid(freq)
    p = pts
    total, amp, scale, norm = torch.zeros(p.shape[:2], dtype=torch.float64, device="cuda"), 1.0, 4.0, 0.0
    for _ in range(6):
        for _ in range(3):
            k = torch.randn(3, generator=g, device="cuda", dtype=torch.float64)
            ph = torch.rand(1, generator=g, device="cuda", dtype=torch.float64) * (2.0 * math.pi)
            total += amp * torch.sin((p @ k) * scale + ph)
        norm += 3.0 * amp
        amp *= 0.5
        scale *= 2.0
    p = p * (1.0 + 0.05 * (2.0 / norm) * total)[..., None]
    t = p[:, local].reshape(-1, 3, 3)
    n = torch.linalg.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    flip = (n * t.mean(1)).sum(1) < 0
    t = torch.where(flip[:, None, None], t[:, [0, 2, 1]], t)
    return t.reshape(-1, 9).float().contiguous()


def _mesh_arrays(freq, seed):
    """The displaced sphere on a ground quad under a sphere light: host vertices, material
    indices and materials (60% Lambert, 25% rough metal, 15% glass, by triangle)."""
    sphere = _sphere(freq, _gen(seed)).cpu().numpy()
    a, b, c, d = [(x, -1.1, z) for x, z in ((-12, -12), (-12, 12), (12, 12), (12, -12))]
    ground = np.array([a + b + c, a + c + d], np.float32)
    light = (scenes.geodesic_sphere(8) * 0.5 + np.array([2.5, 3.0, -1.5])).reshape(-1, 9).astype(np.float32)
    r = np.random.default_rng(seed)
    rows = [{"colour": tuple(r.uniform(0.1, 0.9, 3)) + (1.0,)} for _ in range(614)]
    rows += [{"shade_type": _abi.SHADE_METAL, "roughness": float(r.uniform(0.05, 0.5)),
              "colour": tuple(r.uniform(0.5, 1.0, 3)) + (1.0,)} for _ in range(256)]
    rows += [{"shade_type": _abi.SHADE_GLASS, "ior": 1.5} for _ in range(154)]
    rows += [{"colour": (0.5, 0.5, 0.5, 1.0)}, {"colour": (1.0, 0.95, 0.9, 1.0), "emission": 20.0}]
    u, pick = r.random(len(sphere)), r.random(len(sphere))
    first = np.where(u < 0.6, 0, np.where(u < 0.85, 614, 870))
    count = np.where(u < 0.6, 614, np.where(u < 0.85, 256, 154))
    idx = np.concatenate([first + (pick * count).astype(np.int64), np.full(2, 1024), np.full(len(light), 1025)])
    return np.concatenate([sphere, ground, light]), idx.astype(np.uint32), scenes.material_table(rows)


def _mesh_scene(freq, seed, width=8, leaf=1):
    s = api.Scene(context(), *_mesh_arrays(freq, seed))
    s.set_skybox(np.ones((1, 1, 4), np.float32))
    return s.build(width, 1, leaf)


def _box_scene(width=8, leaf=3):
    b = scenes.box_scene()
    return api.Scene(context(), b["verts"], b["mat_idx"], b["mats"]).build(width, 1, leaf)


def _orbit(r, box):
    """A camera on the orbit of the batched views: an arc before the open box, or around the mesh."""
    a = r.uniform(-25.0, 25.0) if box else r.uniform(-180.0, 180.0)
    b = r.uniform(-6.0, 6.0) if box else r.uniform(-20.0, 10.0)
    ra, rb = math.radians(a), math.radians(b)
    fwd = np.array([math.sin(ra) * math.cos(rb), -math.sin(rb), math.cos(ra) * math.cos(rb)])
    pos = np.array([0.5, 0.5, 0.5]) - 1.9 * fwd if box else -3.4 * fwd
    return dict(position=tuple(pos), rotation=(a, b, 0.0), fov=40.0 if box else 45.0)


def _rays(n, seed, centre, radius, spread, shadow=False):
    """float32 [n, 8] crg_ray records from a sphere around `centre` towards points of a cube of
    half-width `spread` about it."""
    g = _gen(seed)
    rays = torch.empty(n, 8, device="cuda")
    step = 1 << 22
    for at in range(0, n, step):
        m = min(step, n - at)
        o = torch.randn(m, 3, generator=g, device="cuda", dtype=torch.float64)
        o = centre + o / o.norm(dim=1, keepdim=True) * radius
        d = centre + (torch.rand(m, 3, generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0) * spread - o
        d /= d.norm(dim=1, keepdim=True)
        r = rays[at:at + m]
        r[:, 0:3], r[:, 4:7] = o.float(), d.float()
        r[:, 3] = 1e-5
        r[:, 7] = (0.1 + 0.9 * torch.rand(m, generator=g, device="cuda")) if shadow else math.inf
    return rays


def _hit_views(hits):
    w = hits.view(torch.int32)
    return {"t": hits[:, 0], "prim": w[:, 1], "u": hits[:, 2], "v": hits[:, 3]}


def _film(st, w, h, f64=False):
    f = st.own(api.Film(context(), w, h, f64=f64))
    held = st.held[-1]
    p, p64, q64 = C.c_void_p(), C.c_void_p(), C.c_void_p()
    context().check(context().lib.crg_film_device_ptrs(f.h, C.byref(p), C.byref(p64), C.byref(q64)))
    out = {"sum": _tensor(held, p.value, (h, w, 3), torch.float32)}
    if f64:
        out["sum64"] = _tensor(held, p64.value, (h, w, 3), torch.float64)
        out["sumsq64"] = _tensor(held, q64.value, (h, w, 3), torch.float64)
    return f, out


def _buffer(st, shape, dtype):
    b = st.own(api.DeviceBuffer(context(), math.prod(shape) * (8 if dtype == torch.float64 else 4)))
    return b, _tensor(st.held[-1], b.ptr.value, shape, dtype)


def _image(st, w, h):
    return _buffer(st, (h, w, 4), torch.float32)


# ----------------------------------------------------------------------------- cases
SIZES = [(128, 128), (256, 256), (512, 512), (1024, 768), (1920, 1080)]  # the batched views' resolutions


def listed():
    return [
        # a click in the viewport: the smallest call, all latency
        dict(name="pick", kind="pick", rays=127, freq=24),
        # the traversal benchmark: incoherent closest hits, 1,048,576 triangles
        dict(name="closest_soup", kind="closest", rays=1 << 24, tris=1 << 20, width=8),
        # its shadow rays, an odd count (the tail of a larger set)
        dict(name="any_soup", kind="any", rays=5000003, tris=1 << 20, width=8),
        # the plain path tracer on the box: 512x512, 64 spp, depth 8, roulette after 3
        dict(name="render_box", kind="render", scene="box", freq=0, w=512, h=512, spp=64, bounces=8, rr=3, mode=1, f64=False),
        # a progressive pass over the largest mesh: 1920x1080, 4 of its 256 spp, depth 16
        dict(name="render_mesh", kind="render", scene="mesh", freq=458, w=1920, h=1080, spp=4, bounces=16, rr=3, mode=1, f64=False),
        # the reference estimator in the viewport: instances, sun, image sky, odd window
        dict(name="viewport", kind="viewport", w=1283, h=721, spp=1, bounces=5),
        # the smallest batch (a thumbnail): latency and launches
        dict(name="batch_thumb", kind="batch", views=1, mix=0, cap=4096, freq=0, wait=True),
        # views of uneven resolution and spp over both scenes in one launch
        dict(name="batch_views", kind="batch", views=10, mix=7, cap=400000000, freq=458, wait=True),
        # inverse rendering: 256x256, 32 spp forward, 32 spp adjoint
        dict(name="inverse_step", kind="inverse", w=256, h=256, spp=32),
        # bloom and filmic tone curve on a finished 4K frame
        dict(name="post_4k", kind="post", w=3840, h=2160, bloom=True, gray=False, tone=3, full=True),
        # the largest mesh rebuilt under two candidate options, then queried
        dict(name="rebuild_mesh", kind="rebuild", freq=458, width=8),
        # an animated mesh, built anew each frame by a host that owns the GPU's memory
        dict(name="dynamic_mesh", kind="dynamic", tris=10007, width=8, leaf=3, treelet=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pick", "closest", "any", "render", "viewport", "batch", "inverse", "post", "rebuild", "dynamic"])
    c = dict(kind=kind)
    if kind == "pick":
        c.update(rays=_log(rng, 1, 4096), freq=_log(rng, 4, 64))
    elif kind in ("closest", "any"):
        c.update(rays=_log(rng, 1 << 16, 1 << 24), tris=_log(rng, 1 << 12, 1 << 20), width=rng.choice([8, 8, 8, 4, 2]))
    elif kind == "render":
        box = rng.random() < 0.5
        w, h = _log(rng, 65, 1920), _log(rng, 65, 1080)
        c.update(scene="box" if box else "mesh", freq=0 if box else _log(rng, 16, 458), w=w, h=h,
                 spp=max(1, min(_log(rng, 1, 256), (1 << 25) // (w * h))), bounces=8 if box else 16,
                 rr=rng.choice([0, 3]), mode=rng.choice([1, 1, 0]), f64=rng.random() < 0.3)
    elif kind == "viewport":
        c.update(w=_log(rng, 320, 1920), h=_log(rng, 240, 1080), spp=rng.choice([1, 2, 4]), bounces=rng.choice([3, 5, 8]))
    elif kind == "batch":
        c.update(views=rng.randint(1, 10), mix=rng.randint(1, 1 << 20), cap=_log(rng, 4096, 300000000),
                 freq=_log(rng, 16, 458), wait=True)
    elif kind == "inverse":
        c.update(w=_log(rng, 64, 384), h=_log(rng, 64, 384), spp=_log(rng, 4, 64))
    elif kind == "post":
        c.update(w=_log(rng, 200, 3840), h=_log(rng, 150, 2160), bloom=rng.random() < 0.75, gray=rng.random() < 0.3,
                 tone=rng.randint(0, 3), full=rng.random() < 0.5)
    elif kind == "rebuild":
        c.update(freq=_log(rng, 8, 458), width=rng.choice([8, 8, 4, 2]))
    else:
        c.update(tris=_log(rng, 2, 16384), width=rng.choice([8, 8, 4, 2]), leaf=rng.randint(1, 3), treelet=rng.randint(0, 1))
    return c


def _views(case):
    """(box?, width, height, spp) of every view of a batch: drawn by `mix` from the batched
    workload's resolutions and spp, the largest halved until `cap` samples are not exceeded."""
    if case["views"] == 1 and case["cap"] <= 4096:
        return [(True, 64, 64, 1)]
    r = np.random.default_rng(case["mix"])
    v = []
    for _ in range(case["views"]):
        w, h = SIZES[int(r.integers(5))]
        v.append([bool(r.integers(2)), w, h, [16, 64, 256][int(r.integers(3))]])
    while sum(w * h * s for _, w, h, s in v) > case["cap"]:
        k = max(range(len(v)), key=lambda i: v[i][1] * v[i][2] * v[i][3])
        if v[k][3] > 1:
            v[k][3] //= 2
        elif v[k][1] > 64:
            v[k][1:3] = [max(64, v[k][1] * 5 // 8), max(48, v[k][2] * 5 // 8)]
        elif len(v) > 1:
            v.pop(k)
        else:
            break
    return [tuple(x) for x in v]


def prepare(case, seed):
    st = State(case["kind"])
    ctx, kind = context(), case["kind"]
    r = np.random.default_rng(seed)
    if kind == "pick":
        verts = _sphere(case["freq"], _gen(seed)).cpu().numpy()
        st.scene = st.own(api.Scene(ctx, verts, np.zeros(len(verts), np.uint32), scenes.material_table([{}])).build())
        st.rays = _rays(case["rays"], seed + 1, 0.0, 3.4, 0.7)
        st.hits = torch.zeros(case["rays"], 4, device="cuda")
        st.out = _hit_views(st.hits)
    elif kind in ("closest", "any"):
        g = _gen(seed)
        verts = (torch.rand(case["tris"], 1, 3, generator=g, device="cuda", dtype=torch.float64)
                 + 0.01 * torch.randn(case["tris"], 3, 3, generator=g, device="cuda", dtype=torch.float64))
        verts = verts.reshape(-1, 9).float().cpu().numpy()
        st.scene = st.own(api.Scene(ctx, verts, np.zeros(len(verts), np.uint32), scenes.material_table([{}])).build(case["width"]))
        st.rays = _rays(case["rays"], seed + 1, 0.5, math.sqrt(3.0) / 2.0, 0.5, shadow=kind == "any")
        if kind == "closest":
            st.hits = torch.zeros(case["rays"], 4, device="cuda")
            st.out = _hit_views(st.hits)
        else:
            st.occ = torch.zeros(case["rays"], dtype=torch.int32, device="cuda")
    elif kind == "render":
        box = case["scene"] == "box"
        st.scene = st.own(_box_scene() if box else _mesh_scene(case["freq"], seed))
        st.cam = _orbit(r, box)
        st.set = api.make_settings(case["w"], case["h"], case["spp"], case["bounces"], case["rr"], case["mode"], seed,
                                   case["w"] / case["h"])
        st.film, st.out = _film(st, case["w"], case["h"], case["f64"])
    elif kind == "viewport":
        m = scenes.multi_model_box()
        st.scene = st.own(api.Scene.from_models(ctx, m))
        sky = np.ones((256, 512, 4), np.float32)
        sky[..., :3] = r.uniform(0.2, 1.0, (256, 512, 3))
        st.scene.set_skybox(sky, (0.25, 0.0))
        st.scene.set_sun(True)
        st.scene.build()
        st.cam = _orbit(r, True)
        st.set = api.make_settings(case["w"], case["h"], case["spp"], case["bounces"], 0, 0, seed, case["w"] / case["h"])
        st.film, film_out = _film(st, case["w"], case["h"])
        st.image, img = _image(st, case["w"], case["h"])
        st.out = dict(film_out, image=img)
    elif kind == "batch":
        views = _views(case)
        use = sorted({b for b, _, _, _ in views}, reverse=True)
        st.scenes = [st.own(_box_scene() if b else _mesh_scene(max(case["freq"], 16), seed)) for b in use]
        st.views, st.films, st.out = [], [], []
        for k, (b, w, h, spp) in enumerate(views):
            s = api.make_settings(w, h, spp, 8 if b else 16, 3, 1, seed + 31 * k, w / h)
            st.views.append((use.index(b), _orbit(r, b), s))
            f, o = _film(st, w, h)
            st.films.append(f)
            st.out.append(o["sum"])
    elif kind == "inverse":
        w, h, spp = case["w"], case["h"], case["spp"]
        true = scenes.inverse_box()
        sc = st.own(api.Scene(ctx, true["verts"], true["mat_idx"], true["mats"]).build())
        target, t = _film(st, w, h)
        api.render(sc, true["camera"], api.make_settings(w, h, 256, 8, 3, 1, seed + 5), target)
        st.target, t256 = _buffer(st, (h, w, 3), torch.float32)
        t256.copy_(t["sum"] / 256.0)
        start = scenes.inverse_box(r.uniform(0.3, 0.7, (34, 3)), r.uniform(0.4, 0.8, 3))
        st.scene = st.own(api.Scene(ctx, start["verts"], start["mat_idx"], start["mats"]).build())
        st.cam = true["camera"]
        st.fwd = api.make_settings(w, h, spp, 8, 3, 1, seed + 1)
        st.bwd = api.make_settings(w, h, spp, 8, 3, 1, seed + 2)
        st.film, film_out = _film(st, w, h)
        nmat = len(start["mats"])
        shapes = [((h, w, 3), torch.float32), ((1,), torch.float64), ((nmat, 3), torch.float64), ((nmat,), torch.float64)]
        st.bufs, (st.adj, st.loss, st.g_col, st.g_em) = zip(*[_buffer(st, *x) for x in shapes])
        st.out = dict(film_out, adjoint=st.adj, loss=st.loss, g_colour=st.g_col, g_emission=st.g_em)
    elif kind == "post":
        w, h = case["w"], case["h"]
        st.src, src = _image(st, w, h)
        src.copy_(_post_image(case, seed))
        st.dst, st.out = _image(st, w, h)
        st.set = api.post_settings(bloom=int(case["bloom"]), gray_scale=int(case["gray"]), tonemapping=1,
                                   tonemap_type=case["tone"], exposure=1.5, mode=int(case["full"]))
        st.size = (w, h)
    elif kind == "rebuild":
        st.scene = st.own(api.Scene(ctx, *_mesh_arrays(case["freq"], seed)))
        st.rays = _rays(65536, seed + 1, 0.0, 3.4, 0.9)
        st.hits = [torch.zeros(65536, 4, device="cuda") for _ in range(2)]
        st.width = case["width"]
        st.out = [_hit_views(h) for h in st.hits]
    else:
        n = case["tris"]
        g = _gen(seed)
        freq = max(1, math.ceil(math.sqrt(n / 20.0)))
        st.verts = _sphere(freq, g)[torch.randperm(20 * freq * freq, generator=g, device="cuda")[:n]].contiguous()
        st.opts = _abi.BuildOpts(case["width"], case["treelet"], case["leaf"], 3)
        st.info = _abi.BvhInfo()
        node = {8: 80, 4: 64, 2: 48}[case["width"]]
        st.wide = torch.zeros(max(1, n - 1) * node // 4, dtype=torch.int32, device="cuda")
        st.tris = torch.zeros(n, 12, dtype=torch.int32, device="cuda")
        st.order = torch.zeros(n, dtype=torch.int32, device="cuda")
        st.out = dict(wide=st.wide, tris=st.tris, order=st.order)
    torch.cuda.synchronize()
    return st


def run(st):
    ctx, kind = context(), st.kind
    lib = ctx.lib
    if kind in ("pick", "closest"):
        ctx.check(lib.crg_intersect_closest(st.scene.h, st.rays.data_ptr(), st.hits.data_ptr(), len(st.rays), None))
        return st.out
    if kind == "any":
        ctx.check(lib.crg_intersect_any(st.scene.h, st.rays.data_ptr(), st.occ.data_ptr(), len(st.rays), None))
        return st.occ
    if kind == "render":
        st.film.reset()
        api.render(st.scene, st.cam, st.set, st.film)
        return st.out
    if kind == "viewport":
        st.film.reset()
        api.render(st.scene, st.cam, st.set, st.film)
        api.film_display(st.film, st.image)
        return st.out
    if kind == "batch":
        for f in st.films:
            f.reset()
        ctx.check(api.render_batch(st.scenes, st.views, st.films))
        return st.out
    if kind == "inverse":
        st.film.reset()
        api.render(st.scene, st.cam, st.fwd, st.film)
        api.loss_l2(st.film, st.target, st.bufs[0], st.bufs[1])
        st.g_col.zero_()
        st.g_em.zero_()
        api.backward(st.scene, st.cam, st.bwd, st.bufs[0], st.bufs[2], st.bufs[3])
        return st.out
    if kind == "post":
        api.post_process(ctx, st.src, st.dst, *st.size, st.set)
        return st.out
    if kind == "rebuild":
        for k, (treelet, leaf) in enumerate(((0, 3), (1, 1))):  # the default options, then the batched views' best
            st.scene.build(st.width, treelet, leaf)
            ctx.check(lib.crg_intersect_closest(st.scene.h, st.rays.data_ptr(), st.hits[k].data_ptr(), len(st.rays), None))
        return st.out
    ctx.check(lib.crg_build_bvh_noalloc(st.verts.data_ptr(), len(st.verts), C.byref(st.opts), st.wide.data_ptr(),
                                        st.wide.numel() * 4, st.tris.data_ptr(), st.order.data_ptr(), C.byref(st.info), None))
    return st.out


def work(case):
    """Inputs read once and outputs written once; operations: two traversals' node and triangle
    tests per path segment (a node of eight boxes per level, a few triangles), or the taps of the
    blur, or the keys, boxes and nodes of a build."""
    kind = case["kind"]

    def cast(tris):
        return 100.0 * max(1.0, math.log(max(tris, 8), 8)) + 150.0

    if kind in ("pick", "closest", "any"):
        n, t = case["rays"], case.get("tris") or 20 * case["freq"] ** 2
        return {"bytes": n * (36 if kind == "any" else 48) + 48 * min(t, 64 * n), "flops": n * cast(t)}
    if kind in ("render", "viewport"):
        px = case["w"] * case["h"]
        t = 36 if kind == "viewport" or case["scene"] == "box" else 20 * case["freq"] ** 2 + 1282
        per_px = 28 if kind == "viewport" else 60 if case["f64"] else 12
        return {"bytes": px * per_px + 48 * t, "flops": 2.0 * px * case["spp"] * (2 * cast(t) + 300)}
    if kind == "batch":
        b = f = 0.0
        t = 20 * max(case["freq"], 16) ** 2 + 1282
        for box, w, h, spp in _views(case):
            b += 12 * w * h
            f += 2.0 * w * h * spp * (2 * cast(36 if box else t) + 300)
        return {"bytes": b + 48 * t * any(not v[0] for v in _views(case)), "flops": f}
    if kind == "inverse":
        px = case["w"] * case["h"]
        return {"bytes": px * 36.0, "flops": 4.0 * px * case["spp"] * (2 * cast(36) + 300)}
    if kind == "post":
        px = case["w"] * case["h"]
        return {"bytes": px * 32.0, "flops": px * (900.0 * case["bloom"] + 100.0)}
    t = case["tris"] if kind == "dynamic" else 2 * (20 * case["freq"] ** 2 + 1282)
    return {"bytes": t * (36.0 + 48.0 + 4.0 + 32.0 + 20.0), "flops": t * 1000.0}


# ----------------------------------------------------------------------------- 64-bit values
def _post_image(case, seed):
    """An HDR-like image: mostly dark, some texels far above one."""
    g = _gen(seed)
    u = torch.rand(case["h"], case["w"], 4, generator=g, device="cuda")
    img = 0.6 * u * u + 4.0 * (u > 0.97)
    img[..., 3] = 1.0
    return img


def _exact_pick(case, seed):
    tri = _sphere(case["freq"], _gen(seed)).double().reshape(-1, 3, 3)
    rays = _rays(case["rays"], seed + 1, 0.0, 3.4, 0.7).double()
    t_out, u_out, v_out = [], [], []
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    for r in rays.split(64):
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        p = torch.linalg.cross(d.expand(-1, len(tri), -1), e2[None].expand(len(r), -1, -1))
        det = (e1[None] * p).sum(-1)
        s = o - tri[None, :, 0]
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand(len(r), -1, -1))
        v = (d * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-5)
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, at = t.min(1)
        hit = torch.isfinite(best)
        pick = lambda x: torch.where(hit, x.gather(1, at[:, None])[:, 0], torch.zeros_like(best))  # noqa: E731
        t_out.append(best)
        u_out.append(pick(u))
        v_out.append(pick(v))
    return {"t": torch.cat(t_out), "prim": None, "u": torch.cat(u_out), "v": torch.cat(v_out)}


BLUR = [0.19744746769063704, 0.1746973468158936, 0.12099884565428047, 0.06560233156931679, 0.027839605612666265,
        0.009246250740395456, 0.002403157286908872, 0.00048872837522002]


def _exact_post(case, seed):
    w, h, faithful = case["w"], case["h"], not case["full"]
    src = _post_image(case, seed)
    rw, rh = (w // 8 * 8, h // 8 * 8) if faithful else (w, h)
    cover = torch.zeros(h, w, 1, dtype=torch.bool, device="cuda")
    cover[:rh, :rw] = True
    f = src[..., :3].double()
    if case["bloom"]:
        lum = (src[..., 0] * 0.2126 + src[..., 1] * 0.7152) + src[..., 2] * 0.0722
        dark = lum < 0.7
        if faithful:  # the threshold visits pixel (i % w, i / h) for i < w * h
            i = torch.arange(w * h, device="cuda")
            x, y = i % w, i // h
            seen = torch.zeros(h, w, dtype=torch.bool, device="cuda")
            seen[y[y < h], x[y < h]] = True
            dark &= seen
        b = torch.where(dark[..., None], torch.zeros_like(f), f)
        k = torch.tensor(BLUR, device="cuda").float().double()
        for n in range(10):
            dim = 1 if n % 2 == 0 else 0
            out = b * k[0]
            for i in range(1, 8):
                size = b.shape[dim]
                if i < size:
                    out.narrow(dim, 0, size - i).add_(b.narrow(dim, i, size - i) * k[i])
                    out.narrow(dim, i, size - i).add_(b.narrow(dim, 0, size - i) * k[i])
            b = torch.where(cover, out, torch.zeros_like(out))
        f = f + b
    if case["gray"]:
        f = (0.2126 * f[..., 0:1] + 0.7162 * f[..., 1:2] + 0.0722 * f[..., 2:3]).expand(-1, -1, 3)
    e = f * 1.5
    inv = 1.0 / float(np.float32(2.2))

    def hable(x):
        return ((x * (0.15 * x + 0.05) + 0.004) / (x * (0.15 * x + 0.5) + 0.06)) - 0.02 / 0.3

    if case["tone"] == 0:
        f = e ** inv
    elif case["tone"] == 1:
        f = (e / (e + 1.0)) ** inv
    elif case["tone"] == 2:
        x = (e - 0.004).clamp(min=0.0)
        f = (x * (6.2 * x + 0.5)) / (x * (6.2 * x + 1.7) + 0.06)
    else:
        f = (hable(2.0 * e) / hable(11.2)).clamp(min=0.0) ** inv
    out = torch.cat([f, torch.ones_like(f[..., :1])], -1)
    return torch.where(cover, out, torch.zeros_like(out))


def exact(case, seed):
    """Plain 64-bit values where the outputs are formulas of the inputs: hits by testing every
    triangle, the post-processing chain.  Renders are sums of random paths and have none."""
    if case["kind"] == "pick":
        return _exact_pick(case, seed)
    if case["kind"] == "post":
        return _exact_post(case, seed)
    return None
