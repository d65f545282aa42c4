"""The work that a user has this ray tracer do, as measurable cases.

Every case goes through the C ABI by its Python binding (rtgb.capi), as a
program that embeds the library does: geometry and cameras are at hand, the
scene is uploaded once, and one pass is one call or one frame.  Kinds:

- ``render``     one image of a scene that is already built (a viewer that
                 moves its camera, a thumbnail service);
- ``frame``      new vertices on the device, LBVH rebuild, image: the loop of
                 an animated scene;
- ``host_frame`` the same from pinned host memory to a host image, through
                 rt_render_host;
- ``build``      the LBVH build alone;
- ``refit``      device-side animation, refit and image (the wave demo);
- ``stages``     the frame by the reference's stages (primary rays, trace,
                 shadow trace, shade, secondary rays, framebuffer copy), as a
                 renderer written against the drop-in classes runs it;
- ``instances``  new transforms, then one image of a multi-root scene;
- ``batch``      many scenes built and many images rendered in one graph
                 replay;
- ``served``     a burst of requests to the request loop.

Scenes are the repository's own: triangle soups with 20 % mirrors, and fBm
terrains with mirror (or glass) spheres above them.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "tesina-rt_gb300"))
from rtgb import abi, capi, scenes  # noqa: E402

_CTX = None


def _ctx():
    """The program's one context."""
    global _CTX
    if _CTX is None:
        _CTX = capi.Context(0)
    return _CTX


class _Buf:
    """A torch tensor as the binding's device buffer."""

    def __init__(self, shape, dtype):
        self.t = torch.zeros(shape, dtype=dtype, device="cuda")
        self.ptr = ctypes.c_void_p(self.t.data_ptr())


class _View:
    """Device memory of the library as a torch tensor, which keeps the scene
    that owns the memory alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr.value, False), "shape": shape,
                                         "typestr": "<i4", "version": 3}


# ---------------------------------------------------------------------------
# geometry (on the GPU: the large scenes are made many times)
# ---------------------------------------------------------------------------
def _gen(seed, k=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * int(seed) + k)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _pad(v3):
    return torch.nn.functional.pad(v3, (0, 1))


def _np(t, dtype):
    return np.ascontiguousarray(t.cpu().numpy().view(dtype))


def _materials(rows):
    m = np.zeros(len(rows), dtype=abi.MATERIAL_DTYPE)
    m["texture"] = -1
    for i, (diffuse, refl, index) in enumerate(rows):
        m["diffuse"][i, :3] = diffuse
        m["reflectiveness"][i] = refl
        m["refractive_index"][i] = index
    return m


def _point_lights(n):
    """One light as the soups have it, two as the mid-scale terrain, three as
    the stress terrain."""
    pos = {1: [(0.0, 4.0, -2.0)], 2: [(-4.0, 6.0, -3.0), (5.0, 5.0, 2.0)],
           3: [(-4.0, 6.0, -3.0), (5.0, 5.0, 2.0), (0.0, 8.0, 6.0)]}[n]
    col = {1: [(1.0, 1.0, 1.0)], 2: [(0.7, 0.7, 0.7), (0.5, 0.5, 0.6)],
           3: [(0.6, 0.6, 0.6), (0.4, 0.4, 0.5), (0.3, 0.3, 0.3)]}[n]
    return [dict(type=abi.RT_POINT_L, pos=p, color=c) for p, c in zip(pos, col)]


def _soup(n, seed, lights=1):
    """Triangle soup: centroids uniform in [-1, 1]^3, vertex offsets
    N(0, 0.03), 20 % mirrors of reflectance 0.5, the rest Lambertian."""
    g = _gen(seed)
    c = _rand(g, n, 1, 3) * 2 - 1
    v = c + torch.randn(n, 3, 3, generator=g, device="cuda") * 0.03
    fn = torch.nn.functional.normalize(torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]), dim=1)
    pos, nrm = _pad(v.reshape(-1, 3)), _pad(fn.repeat_interleave(3, dim=0))
    mirror = _rand(g, n) < 0.2
    mats = np.zeros(n + 1, dtype=abi.MATERIAL_DTYPE)
    mats["texture"] = -1
    mats["reflectiveness"][0] = 0.5
    mats["diffuse"][1:, :3] = (_rand(g, n, 3) * 0.7 + 0.2).cpu().numpy()
    slots = torch.arange(1, n + 1, device="cuda", dtype=torch.int32)
    mat_map = torch.where(mirror, torch.zeros_like(slots), slots)
    idx = torch.arange(3 * n, device="cuda", dtype=torch.int32)
    return scenes.Scene(_np(pos, np.float32), _np(nrm, np.float32), _np(idx, np.uint32), mats,
                        _np(mat_map, np.uint32),
                        abi.make_lights((0.1,) * 3, _point_lights(lights)))


def _terrain(nx, nz, spheres, seed, lights=2, glass=False):
    """fBm height field of nx x nz cells over [-8, 8] x [-4, 4] (four octaves,
    first lattice cell 2 units) with mirror or glass spheres above it."""
    g = _gen(seed, 1)
    h, amp, cells = torch.zeros(nz + 1, nx + 1, device="cuda"), 1.0, 4
    for _ in range(4):
        lattice = _rand(g, 1, 1, cells + 1, 2 * cells + 1) * 2 - 1
        h += amp * torch.nn.functional.interpolate(lattice, size=(nz + 1, nx + 1), mode="bicubic",
                                                   align_corners=True)[0, 0]
        amp, cells = amp * 0.5, cells * 2
    xs = torch.linspace(-8, 8, nx + 1, device="cuda")
    zs = torch.linspace(-4, 4, nz + 1, device="cuda")
    gz, gx = torch.meshgrid(zs, xs, indexing="ij")
    dz, dx = torch.gradient(h, spacing=(8.0 / nz, 16.0 / nx))
    nrm = torch.nn.functional.normalize(torch.stack([-dx, torch.ones_like(h), -dz], -1).reshape(-1, 3), dim=1)
    pos = torch.stack([gx, h, gz], -1).reshape(-1, 3)
    j, i = torch.meshgrid(torch.arange(nz, device="cuda"), torch.arange(nx, device="cuda"), indexing="ij")
    v00 = (j * (nx + 1) + i).reshape(-1)
    v01 = v00 + nx + 1
    tris = torch.stack([v00, v00 + 1, v01 + 1, v00, v01 + 1, v01], 1).reshape(-1, 3)
    # UV spheres of 32 x 16 segments, 960 triangles each
    seg, rings = 32, 16
    th = torch.arange(1, rings, device="cuda").float().mul(math.pi / rings)[:, None]
    ph = torch.arange(seg, device="cuda").float().mul(2 * math.pi / seg)[None]
    ring = torch.stack([th.sin() * ph.cos(), th.cos().expand(-1, seg), th.sin() * ph.sin()], -1)
    pole = torch.tensor([[0.0, 1.0, 0.0]], device="cuda")
    unit = torch.cat([pole, ring.reshape(-1, 3), -pole])
    s = torch.arange(seg, device="cuda")
    s1, last = (s + 1) % seg, 1 + (rings - 1) * seg
    st = [torch.stack([torch.zeros_like(s), 1 + s, 1 + s1], 1)]
    for r in range(rings - 2):
        a, b = 1 + r * seg, 1 + (r + 1) * seg
        st += [torch.stack([a + s, b + s, b + s1], 1), torch.stack([a + s, b + s1, a + s1], 1)]
    st.append(torch.stack([last - seg + s, torch.full_like(s, last), last - seg + s1], 1))
    st = torch.cat(st)
    rad = _rand(g, spheres, 1) * 0.4 + 0.1
    cen = torch.cat([_rand(g, spheres, 1) * 15 - 7.5, rad + 0.6 + _rand(g, spheres, 1) * 1.6,
                     _rand(g, spheres, 1) * 7 - 3.5], 1)
    sp = (unit[None] * rad[:, None] + cen[:, None]).reshape(-1, 3)
    sn = unit.repeat(spheres, 1)
    stris = (st[None] + (pos.shape[0] + unit.shape[0] * torch.arange(spheres, device="cuda"))[:, None, None])
    idx = torch.cat([tris, stris.reshape(-1, 3)]).to(torch.int32)
    mat_map = torch.zeros(idx.shape[0], dtype=torch.int32, device="cuda")
    mat_map[tris.shape[0]:] = 1
    sphere = ((0.1,) * 3, 0.9, 1.333) if glass else ((0.1,) * 3, 0.8, 0.0)
    return scenes.Scene(_np(_pad(torch.cat([pos, sp])), np.float32),
                        _np(_pad(torch.cat([nrm, sn])), np.float32), _np(idx, np.uint32),
                        _materials([((0.55, 0.5, 0.4), 0.0, 0.0), sphere]), _np(mat_map, np.uint32),
                        abi.make_lights((0.1,) * 3, _point_lights(lights)))


def _scene(case, seed):
    if case["scene"] == "soup":
        return _soup(case["tris"], seed)
    return _terrain(case["nx"], case["nz"], case["spheres"], seed, case.get("lights", 2),
                    case.get("glass", False))


def _tris(case):
    if case["scene"] == "soup":
        return case["tris"]
    return 2 * case["nx"] * case["nz"] + 960 * case["spheres"]


def _camera(case, seed):
    """The workloads' cameras, turned a little by the seed."""
    w, h = case["width"], case["height"]
    r = np.random.default_rng(int(seed))
    j = r.uniform(-0.2, 0.2, 3)
    if case["scene"] == "soup":
        return scenes.camera((j[0], j[1], -4.0 + j[2]), (0.0, 0.0, 0.0), fov_deg=60.0, aspect=w / h)
    if case.get("orbit"):   # a pose on a sphere about the field, above it
        v = np.array([6.0 + 8 * j[0], 5.5 + 8 * j[1], -6.0 + 8 * j[2]])
        v *= 10.0 / np.linalg.norm(v)
        return scenes.camera(tuple(v), (0.0, 0.0, 0.0), fov_deg=60.0, aspect=w / h)
    return scenes.camera((j[0], 9.0 + j[1], -2.5 + j[2]), (0.0, 0.0, 2.0), fov_deg=60.0, aspect=w / h)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    mid = dict(scene="terrain", nx=1024, nz=512, spheres=200)        # 1,240,576 triangles
    stress = dict(scene="terrain", nx=4096, nz=2048, spheres=1000)   # 17,737,216 triangles
    hd = dict(width=1920, height=1080)
    return [
        # a preview tile of a small mesh: the smallest call, launches and latency
        dict(name="thumb_1k", kind="render", scene="soup", tris=1000, width=256, height=256, bounces=1),
        # the small workload as an animated frame: update, rebuild, image
        dict(name="frame_10k", kind="frame", scene="soup", tris=10000, width=512, height=512, bounces=3),
        # LBVH rebuild of the mid-scale mesh (the per-frame rebuild of a game-sized scene)
        dict(name="build_1M", kind="build", **mid),
        # LBVH build of the largest mesh that the workloads name
        dict(name="build_17M", kind="build", **stress),
        # the headline: the mid-scale frame end to end from host buffers
        dict(name="host_frame_1M", kind="host_frame", bounces=4, **mid, **hd),
        # a 4K still of the largest scene, three lights, deep reflections
        dict(name="render_17M_4k", kind="render", bounces=6, width=3840, height=2160, lights=3,
             orbit=True, **stress),
        # the wave demo: the vertices move on the device, the tree is refitted
        dict(name="refit_1M", kind="refit", bounces=4, **mid, **hd),
        # the mid-scale field under glass spheres: reflected and refracted rays
        dict(name="glass_1M", kind="render", bounces=4, glass=True, **mid, **hd),
        # the renderer written against the stage classes, a size that no tile divides
        dict(name="stages_10k", kind="stages", scene="soup", tris=10000, width=1000, height=701, bounces=2),
        # objects with transforms of their own: 4 ground tiles and 12 soups
        dict(name="instances_16", kind="instances", nx=256, nz=128, spheres=20, tris=50000, blobs=12,
             bounces=4, **hd),
        # 64 scenes and images at once (a dataset's renders)
        dict(name="batch_64", kind="batch", count=64, tris_min=1000, tris_max=500000, bounces=4),
        # a burst at the request loop over resident scenes
        dict(name="served_24", kind="served", pool=6, requests=24, tris_min=10000, tris_max=500000,
             bounces=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "frame", "host_frame", "build", "build", "refit", "stages",
                       "instances", "batch", "served"])
    w, h = _log(rng, 96, 2600), _log(rng, 96, 1500)
    b = rng.randint(0, 6)
    if kind == "instances":
        nz = _log(rng, 16, 160)
        return dict(kind=kind, nx=2 * nz, nz=nz, spheres=rng.randint(1, 20), tris=_log(rng, 500, 80000),
                    blobs=rng.randint(1, 30), bounces=rng.randint(0, 5), width=w, height=h)
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 2, 60), tris_min=_log(rng, 300, 3000),
                    tris_max=_log(rng, 10000, 400000), bounces=rng.randint(1, 5))
    if kind == "served":
        return dict(kind=kind, pool=rng.randint(1, 8), requests=rng.randint(1, 30),
                    tris_min=_log(rng, 2000, 20000), tris_max=_log(rng, 30000, 500000),
                    bounces=rng.randint(1, 5))
    if rng.random() < 0.4 and kind != "refit":
        s = dict(scene="soup", tris=_log(rng, 300, 3_000_000 if kind == "build" else 500_000))
    else:
        nz = _log(rng, 12, 1700 if kind == "build" else 800)
        s = dict(scene="terrain", nx=max(8, int(nz * rng.uniform(1.0, 2.4))), nz=nz,
                 spheres=rng.randint(1, 300))
    if kind == "build":
        return dict(kind=kind, **s)
    if kind == "stages":
        w, h = min(w, 1400), min(h, 900)
        b = min(b, 4)
    if kind == "render" and s["scene"] == "terrain" and rng.random() < 0.3:
        s["glass"] = True
        b = min(b, 4)
    if s["scene"] == "terrain":
        s["lights"] = rng.randint(1, 3)
    return dict(kind=kind, width=w, height=h, bounces=b, **s)


_SIZES = [(256, 256), (512, 512), (1024, 768), (333, 257)]


def _batch_items(case, seed):
    """(triangles, width, height, bounces) of each image of a batch or burst:
    triangles log-uniform, so few scenes are large."""
    n = case["count"] if case["kind"] == "batch" else case["pool"]
    r = np.random.default_rng(17 + n)   # the mix belongs to the case, the scenes to the seed
    tri = np.exp(r.uniform(math.log(case["tris_min"]), math.log(case["tris_max"]), n)).round().astype(int)
    size = r.integers(0, len(_SIZES), max(n, case.get("requests", n)))
    depth = r.integers(1, case["bounces"] + 1, size.shape[0])
    return [int(t) for t in tri], [_SIZES[s] for s in size], [int(d) for d in depth]


def _turns(case, seed):
    r = np.random.default_rng(int(seed) + 5)
    inst, ms, mis = [], [], []
    for x in (-1, 1):
        for z in (-1, 1):
            m, mi = scenes.transform(t=(8.0 * x, 0.0, 4.0 * z))
            inst.append(0), ms.append(m), mis.append(mi)
    for _ in range(case["blobs"]):
        s = float(r.uniform(0.4, 1.0))
        m, mi = scenes.transform(float(r.uniform(0, 360)), (s, s, s),
                                 (float(r.uniform(-12, 12)), float(r.uniform(2, 4)), float(r.uniform(-6, 6))))
        inst.append(1), ms.append(m), mis.append(mi)
    return np.array(inst, np.int32), np.array(ms), np.array(mis)


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    st = dict(case=case, ctx=ctx)
    if kind == "batch":
        tri, size, depth = _batch_items(case, seed)
        items = []
        for k, n in enumerate(tri):
            w, h = size[k]
            cam = _camera(dict(scene="soup", width=w, height=h), seed + k)
            items.append((capi.Scene(ctx, _soup(n, 1000 * seed + k)), cam, w, h, depth[k]))
        b = capi.Batch(ctx)
        b.set(items)
        st.update(batch=b, rgba=_Buf((b.pixels, 4), torch.uint8), stats=_Buf((4,), torch.int64))
        b.capture(st["rgba"], st["stats"])
        return st
    if kind == "served":
        tri, size, depth = _batch_items(case, seed)
        srv = capi.Server(ctx, budget=24 << 30, arena=256 << 20, max_views=256, max_inflight=3)
        ids = [srv.add_scene(_soup(n, 1000 * seed + k) if k % 2 == 0 else
                             _terrain(2 * int((n / 4) ** 0.5), int((n / 4) ** 0.5), 4, 1000 * seed + k))
               for k, n in enumerate(tri)]
        req = []
        for k in range(case["requests"]):
            w, h = size[k]
            s = k % len(ids)
            cam = _camera(dict(scene="soup" if s % 2 == 0 else "terrain", width=w, height=h), seed + k)
            req.append((ids[s], cam, w, h, depth[k]))
        st.update(server=srv, requests=req)
        return st
    if kind == "instances":
        meshes = [capi.Scene(ctx, _terrain(case["nx"], case["nz"], case["spheres"], seed)),
                  capi.Scene(ctx, _soup(case["tris"], seed))]
        for m in meshes:
            m.build(30, 1)
        inst, tr, tri = _turns(case, seed)
        lights = abi.make_lights((0.1,) * 3, _point_lights(2))
        st.update(inst=capi.Instances(ctx, meshes, inst, tr, tri, lights), tr=tr, tr_inv=tri)
        st["cam"] = scenes.camera((0.0, 12.0, -16.0), (0.0, 0.0, 0.0), fov_deg=60.0,
                                  aspect=case["width"] / case["height"])
    else:
        host = _scene(case, seed)
        st["scene"] = sc = capi.Scene(ctx, host)
        if kind == "build":
            return st
        st["cam"] = _camera(case, seed)
        if kind in ("render", "refit", "stages"):
            sc.build(30, 1)
        if kind == "refit":
            st["phase"] = float(np.random.default_rng(int(seed)).uniform(0, 6))
        if kind == "frame":   # the next frame's vertices, made on the device by the program
            pos, nrm = torch.from_numpy(host.pos4).cuda(), torch.from_numpy(host.nrm4).cuda()
            pos[:, 1] += 0.1 * torch.sin(pos[:, 0] + 0.1)
            st.update(pos=pos, nrm=nrm)
        if kind == "host_frame":   # a moved copy of the vertices in pinned memory
            pos = torch.from_numpy(host.pos4).clone()
            pos[:, 1] += 0.1 * torch.sin(pos[:, 0] + 0.1)
            st["keep"] = [pos.pin_memory(), torch.from_numpy(host.nrm4).pin_memory(),
                          torch.zeros(case["width"] * case["height"], 4, dtype=torch.uint8).pin_memory()]
            st["pos"], st["nrm"], st["rgba"] = [t.numpy() for t in st["keep"]]
            return st
    px = case["width"] * case["height"]
    st.update(rgba=_Buf((px, 4), torch.uint8), img=_Buf((px, 3), torch.int32),
              stats=_Buf((4,), torch.int64))
    if kind == "stages":
        st["samples"] = [_Buf((px, 20), torch.float32) for _ in range(2)]
        st["hits"] = [_Buf((px, 16), torch.float32) for _ in range(case["bounces"] + 1)]
        st["count"] = _Buf((1,), torch.int32)
    torch.cuda.synchronize()
    return st


def _run_stages(st, case):
    """Renderer::render_to_framebuffer's loop over the stage entry points."""
    ctx, sc = st["ctx"], st["scene"]
    w, h = case["width"], case["height"]
    capi.check(ctx.lib, ctx.lib.rt_fb_clear(ctx.h, st["img"].ptr, w * h, None))
    a, b = st["samples"]
    ctx.gen_primary(st["cam"], w, h, a)
    n = w * h
    counts = []
    for k in range(case["bounces"] + 1):
        hits = st["hits"][k]
        counts.append(n)
        sc.trace(a, n, hits)
        sc.shadow(a, n, hits)
        sc.shade(a, hits, n, st["img"], primary=int(k == 0))
        if k < case["bounces"]:
            n = sc.gen_secondary(a, n, hits, b, w * h, st["count"])
            if n == 0:
                break
            a, b = b, a
    ctx.fb_copy(st["img"], st["rgba"], w * h)
    first = st["hits"][0].t
    counts += [0] * (case["bounces"] + 1 - len(counts))
    return {"rgba": st["rgba"].t, "image": st["img"].t, "rays": np.array(counts),
            "flags": first[:, :1].view(torch.uint8), "t": first[:, 1], "id": first[:, 2].view(torch.int32),
            "normal": first[:, 8:11], "point": first[:, 12:15],
            "last": st["hits"][-1].t.view(torch.uint8)}


def run(state):
    st, ctx = state, state["ctx"]
    case = st["case"]
    kind = case["kind"]
    if kind == "build":
        sc = st["scene"]
        sc.build(30, 1)
        idx, mp, _, _, n = sc.buffers()
        return {"indices": torch.as_tensor(_View(sc, idx, (n, 3)), device="cuda"),
                "material_map": torch.as_tensor(_View(sc, mp, (n,)), device="cuda")}
    if kind == "batch":
        st["batch"].replay()
        return {"rgba": st["rgba"].t, "rays": st["stats"].t}
    if kind == "served":
        srv = st["server"]
        tickets = [srv.submit_render(s, cam, w, h, d) for s, cam, w, h, d in st["requests"]]
        return [srv.result(t, w, h)[0] for t, (_, _, w, h, _) in zip(tickets, st["requests"])]
    w, h, b = case["width"], case["height"], case["bounces"]
    if kind == "host_frame":
        rgba, rays = st["scene"].render_host(st["cam"], w, h, b, st["pos"], st["nrm"], rgba=st["rgba"])
        return {"rgba": rgba, "rays": [rays.primary_rays, rays.secondary_rays, rays.shadow_rays, rays.hits]}
    if kind == "stages":
        return _run_stages(st, case)
    if kind == "instances":
        st["inst"].set_transforms(st["tr"], st["tr_inv"])
        st["inst"].render(st["cam"], w, h, b, st["rgba"], st["img"])
        return {"rgba": st["rgba"].t, "image": st["img"].t}
    sc = st["scene"]
    if kind == "frame":
        p, n = ctypes.c_void_p(st["pos"].data_ptr()), ctypes.c_void_p(st["nrm"].data_ptr())
        capi.check(ctx.lib, ctx.lib.rt_scene_update_vertices_device(ctx.h, sc.h, p, n, st["pos"].shape[0], None))
        sc.build(30, 1)
    elif kind == "refit":
        sc.mangle(st["phase"])
        sc.refit()
    sc.render(st["cam"], w, h, b, st["rgba"], st["img"])
    return {"rgba": st["rgba"].t, "image": st["img"].t}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _build_bytes(n, v):
    """Vertices once; index triple, material and id of each triangle in and,
    in sorted order, out; half as many interior nodes as triangles, two child
    boxes and references each; the triangle's vertices beside the tree."""
    return 16 * v + 40 * n + 32 * n + 36 * n


def _image_work(n, px, lights, hit=0.7):
    """One closest-hit ray per pixel and one shadow ray per light and hit: a
    root-to-leaf path of two box tests per level (2 x 21 operations) and one
    triangle test (50) each; of the scene what that many rays can touch."""
    rays = px * (1 + hit * lights)
    return (16 * px + 80 * min(n, 2 * px),
            rays * (42 * math.log2(max(n, 2)) + 50))


def work(case):
    kind = case["kind"]
    if kind in ("batch", "served"):
        tri, size, _ = _batch_items(case, 0)
        images = len(tri) if kind == "batch" else case["requests"]
        parts = [_image_work(tri[k % len(tri)], size[k][0] * size[k][1], 1, 0.5) for k in range(images)]
        by, fl = (sum(p[i] for p in parts) for i in (0, 1))
        if kind == "batch":
            by += sum(_build_bytes(n, 3 * n) for n in tri)
        return {"bytes": by, "flops": fl}
    if kind == "instances":
        n = 2 * case["nx"] * case["nz"] + 960 * case["spheres"] + case["tris"]
        by, fl = _image_work(n, case["width"] * case["height"], 2)
        return {"bytes": by, "flops": fl}
    n = _tris(case)
    v = 3 * n if case["scene"] == "soup" else (case["nx"] + 1) * (case["nz"] + 1) + 482 * case["spheres"]
    by = fl = 0
    if kind in ("frame", "host_frame", "build"):
        by += _build_bytes(n, v)
    if kind in ("frame", "host_frame", "refit"):
        by += 64 * v   # new vertices read and written
    if kind == "refit":
        by += 12 * n + 16 * v + 32 * n + 36 * n
    if kind != "build":
        i, f = _image_work(n, case["width"] * case["height"], 1 if case["scene"] == "soup" else case.get("lights", 2))
        by, fl = by + i, fl + f
    if kind == "build":
        fl += 60 * n
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------
# the first hits of the stage pipeline in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    """Distance, point and normal of each first hit by brute force over all
    triangles.  Images, ids and flags are whole numbers, and the trees' sorted
    buffers too: they have no value of this kind."""
    if case["kind"] != "stages" or case["scene"] != "soup":
        return None
    w, h, n = case["width"], case["height"], case["tris"]
    if w * h * n > 1e10:
        return None
    sc, cam = _scene(case, seed), _camera(case, seed)
    f8 = lambda a: torch.as_tensor(np.array(a), dtype=torch.float64, device="cuda")  # noqa: E731
    o, cd, cr, cu = [f8(list(getattr(cam, k))[:3]) for k in ("pos", "dir", "right", "up")]
    v = f8(sc.pos4[:, :3])[torch.from_numpy(sc.idx.astype(np.int64)).cuda()]
    nv = f8(sc.nrm4[:, :3])[torch.from_numpy(sc.idx.astype(np.int64)).cuda()]
    # pixel of each ray: 32 x 32 blocks, then the columns right of them, then the rows below
    xb, yb = w // 32, h // 32
    xs, ys = [], []
    if xb and yb:
        b, p = torch.meshgrid(torch.arange(xb * yb), torch.arange(1024), indexing="ij")
        xs.append(((b % xb) * 32 + p % 32).reshape(-1)), ys.append((torch.div(b, xb, rounding_mode="floor") * 32 + p // 32).reshape(-1))
    if w > xb * 32:
        i = torch.arange((w - xb * 32) * h)
        xs.append(xb * 32 + i % (w - xb * 32)), ys.append(i // (w - xb * 32))
    if h > yb * 32:
        i = torch.arange(xb * 32 * (h - yb * 32))
        xs.append(i // (h - yb * 32)), ys.append(yb * 32 + i % (h - yb * 32))
    x, y = torch.cat(xs).cuda().double(), torch.cat(ys).cuda().double()
    d = cd + (2 * (x + 0.5) / w - 1)[:, None] * cr + (2 * (y + 0.5) / h - 1)[:, None] * cu
    d = d / d.norm(dim=1, keepdim=True)
    e1, e2, s = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0], o - v[:, 0]
    q = torch.linalg.cross(s, e1)
    # det = d . (e2 x e1)..., all as products of the ray directions with per-triangle vectors
    nx, su, tq = torch.linalg.cross(e2, e1), torch.linalg.cross(e2, s), (e2 * q).sum(1)
    best = torch.full((d.shape[0],), math.inf, dtype=torch.float64, device="cuda")
    bu, bv = torch.zeros_like(best), torch.zeros_like(best)
    bi = torch.zeros(d.shape[0], dtype=torch.int64, device="cuda")
    step = max(1, 300_000_000 // n)
    for r in range(0, d.shape[0], step):
        dd = d[r:r + step]
        det = dd @ nx.T
        u = (dd @ su.T) / det
        vv = (dd @ q.T) / det
        t = tq / det
        t = torch.where((u < 0) | (vv < 0) | (u + vv > 1) | (t < 0) | ~torch.isfinite(t), math.inf, t)
        m, i = t.min(1)
        best[r:r + step], bi[r:r + step] = m, i
        bu[r:r + step], bv[r:r + step] = u.gather(1, i[:, None])[:, 0], vv.gather(1, i[:, None])[:, 0]
        del det, u, vv, t
    hit = torch.isfinite(best)
    unit = nv / nv.norm(dim=2, keepdim=True)
    nn = unit[bi, 0] * (1 - bu - bv)[:, None] + unit[bi, 1] * bu[:, None] + unit[bi, 2] * bv[:, None]
    nn = nn / nn.norm(dim=1, keepdim=True)
    nn = torch.where((nn * d).sum(1, keepdim=True) > 0, -nn, nn)
    z = torch.zeros((), dtype=torch.float64, device="cuda")
    return {"rgba": None, "image": None, "rays": None, "flags": None, "id": None, "last": None,
            "t": torch.where(hit, best, z), "normal": torch.where(hit[:, None], nn, z),
            "point": torch.where(hit[:, None], o + d * torch.where(hit, best, z)[:, None], z)}
