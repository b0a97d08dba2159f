"""The workloads this renderer's speed is judged on, each run through the
public binding (`prt.Context`) the way an application calls it.

A case is a dict of plain values.  `prepare` makes what an application holds
before the call (scene, acceleration structure, camera, frame, ray buffers),
`run` is one call sequence, `work` the bytes and operations it cannot do
without, and `exact` the same results in 64-bit torch arithmetic (a triangle
search over boxes of consecutive triangles, the documented camera, RNG and
bounce formulas).

Kinds:
  frame    prt_render into the accumulation buffer, which is then read on the device
  viewer   one more pass into the accumulated frame, which is read on the device after each (the reference's render loop)
  train    one optimisation step of per-triangle albedo and sky: render, image loss, adjoint
  batch    prt_render_batch over requests of uneven size and scene
  closest  prt_intersect of incoherent rays
  occluded prt_occluded of short rays (ambient occlusion, shadows)
  rebuild  prt_build_accel on the loaded mesh, then closest hits through the new tree
  mesh     prt_build_mesh of a host triangle soup, then the indexed mesh on the host
"""

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "embree-benchmark-protoray_b200"))

import prt  # noqa: E402
import scenes  # noqa: E402

FLT_MAX = 3.4028234663852886e38
# triangles of the generated scenes, for work(): small, terrain, the sphere field and the batch scenes 0..7
TRIANGLES = {"small": 81922, "terrain": 1376256, "field": 10240000, "batch0": 10242, "batch1": 31556,
             "batch2": 46082, "batch3": 106960, "batch4": 207362, "batch5": 449808, "batch6": 938242,
             "batch7": 2009636}


def listed():
    return [
        # a picking or placement tool: a thousand rays, where launch and host latency are everything
        dict(name="closest_1k_small", kind="closest", scene="small", rays=1000),
        # lidar- or probe-style bulk queries through the intersector seam, incoherent, larger than L2
        dict(name="closest_4m_terrain", kind="closest", scene="terrain", rays=4194304),
        # a bake of short occlusion rays, ragged count
        dict(name="occluded_1m_terrain", kind="occluded", scene="terrain", rays=1000003, reach=0.05),
        # a small preview frame: 256x256, 16 passes, 82K triangles
        dict(name="frame_256_16spp_small", kind="frame", scene="small", width=256, height=256, spp=16, depth=5,
             integrator="diffuse", albedo=False, lens=False, packets=0, wave=0),
        # the reference's interactive loop: one pass per call at 1080p, the refined image shown after each
        dict(name="viewer_hd_terrain", kind="viewer", scene="terrain", width=1920, height=1080, depth=5),
        # the headline frame: 1080p, 64 passes, 1.38M triangles, in the launch configuration its autotuner finds
        dict(name="frame_hd_64spp_terrain", kind="frame", scene="terrain", width=1920, height=1080, spp=64, depth=5,
             integrator="diffuse", albedo=False, lens=False, packets=2, wave=16),
        # the largest scene: 10.24M triangles, 8 bounces, default launch configuration
        dict(name="frame_hd_16spp_field", kind="frame", scene="field", width=1920, height=1080, spp=16, depth=8,
             integrator="diffuse", albedo=False, lens=False, packets=0, wave=0),
        # next-event estimation with a thin lens and textured (per-triangle) albedo at a ragged window size
        dict(name="frame_nee_lens_ragged", kind="frame", scene="terrain", width=1001, height=563, spp=16, depth=5,
             integrator="diffuse2", albedo=True, lens=True, packets=0, wave=0),
        # one step of fitting albedo and sky to an image
        dict(name="train_512_16spp_small", kind="train", scene="small", width=512, height=512, spp=16, depth=5),
        # a render server's queue: requests of uneven size, passes and scene in one call
        dict(name="batch_32_requests", kind="batch", requests=32, mix=7),
        # a deformed or edited scene: rebuild the tree of 1.38M triangles and query it
        dict(name="rebuild_terrain", kind="rebuild", scene="terrain", rays=262144, high=True),
        # scene import: soup of 1.38M triangles to an indexed mesh
        dict(name="mesh_terrain", kind="mesh", scene="terrain", normals=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest", "occluded", "frame", "frame", "frame", "viewer", "train", "batch", "rebuild", "mesh"])
    scene = rng.choice(["small", "terrain", "batch%d" % rng.randrange(8)])
    if kind in ("closest", "occluded"):
        case = dict(kind=kind, scene=scene, rays=_log_int(rng, 1000, 4000000))
        return dict(case, reach=round(rng.uniform(0.01, 0.3), 3)) if kind == "occluded" else case
    if kind == "batch":
        return dict(kind=kind, requests=rng.randint(2, 24), mix=rng.randrange(1 << 20))
    if kind == "rebuild":
        return dict(kind=kind, scene=scene, rays=_log_int(rng, 1000, 300000), high=rng.random() < 0.75)
    if kind == "mesh":
        return dict(kind=kind, scene=scene, normals=rng.random() < 0.5)
    width = _log_int(rng, 64, 1920)
    height = max(48, min(1080, int(width * rng.uniform(0.5, 0.8))))
    depth = rng.randint(1, 8)
    if kind == "viewer":
        return dict(kind=kind, scene=scene, width=width, height=height, depth=depth)
    if kind == "train":
        width, height = min(width, 640), min(height, 480)
        return dict(kind=kind, scene=scene, width=width, height=height, spp=_log_int(rng, 1, 16), depth=depth)
    spp = min(_log_int(rng, 1, 64), max(1, 32000000 // (width * height)))
    return dict(kind=kind, scene=scene, width=width, height=height, spp=spp, depth=depth,
                integrator=rng.choice(["diffuse", "diffuse", "diffuse2"]), albedo=rng.random() < 0.3,
                lens=rng.random() < 0.3, packets=rng.choice([0, 1, 2]) if width >= 1280 else 0, wave=0)


# --- inputs ---------------------------------------------------------------

def _scene(name, seed):
    """(Mesh, View) of a scene; the seed moves its spheres and its terrain."""
    if name == "small":
        return scenes.small_scene(seed)
    if name == "terrain":
        return scenes.terrain_scene(seed)
    if name == "field":
        mesh, _ = scenes.spheres10m_scene(seed)
        return mesh, scenes.field_view(mesh)
    return scenes.batch_scene(int(name[5:]), 100 + 8 * seed)


def _context(mesh, high=True):
    ctx = prt.Context(0)
    ctx.load_mesh(mesh.indices, mesh.positions)
    ctx.set_build_quality(high)
    ctx.build()
    return ctx


def _view(case, view):
    if case.get("lens"):
        view.radius = 0.004 * view.focus
    return view


def _rays(case, mesh, seed):
    """Incoherent ray records: origins uniform in the scene's box, directions uniform on the sphere."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo, hi = (torch.from_numpy(np.asarray(b, np.float32)).cuda() for b in mesh.bounds())
    n = case["rays"]
    rays = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    rays[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")
    rays[:, 3] = 0.0
    d = torch.randn((n, 3), generator=g, device="cuda")
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rays[:, 7] = float(case["reach"] * (hi - lo).norm()) if "reach" in case else FLT_MAX
    return rays


def _requests(case):
    """Sizes of a batch's requests: res 128..1024, 1..64 passes (fewer for large frames), scenes 0..5."""
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["requests"]):
        w, h = rng.randint(128, 1024), rng.randint(128, 1024)
        out.append(dict(scene="batch%d" % rng.randrange(6), width=w, height=h, spp=rng.randint(1, 32), depth=5))
    return out


def _soup(case, mesh):
    soup = np.zeros(mesh.tri_count, prt.SOUP_DTYPE)
    soup["v"]["pos"] = mesh.positions[mesh.indices]
    if case["normals"]:
        # smooth shading from the importer on most triangles, none given on the rest
        n = soup["v"]["pos"] - mesh.positions.mean(axis=0)
        n /= np.maximum(np.linalg.norm(n, axis=-1, keepdims=True), 1e-6)
        n[::5] = 0
        soup["v"]["normal"] = n
    soup["matId"] = np.arange(mesh.tri_count) % 3
    return soup


def _train_inputs(case, mesh, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    albedo = 0.2 + 0.6 * torch.rand(mesh.tri_count, generator=g, device="cuda")
    target = 0.3 + 0.6 * torch.rand((case["height"], case["width"], 3), generator=g, device="cuda")
    return albedo, target


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        reqs = _requests(case)
        ctxs = {}
        for q in reqs:
            if q["scene"] not in ctxs:
                mesh, view = _scene(q["scene"], seed)
                ctxs[q["scene"]] = (_context(mesh), view)
        table = []
        for q in reqs:
            ctx, view = ctxs[q["scene"]]
            table.append(dict(scene=ctx, camera=prt.camera_from_view(view, q["width"], q["height"]), width=q["width"],
                              height=q["height"], spp=q["spp"], maxDepth=q["depth"],
                              accum=torch.empty((q["height"], q["width"], 4), dtype=torch.float32, device="cuda")))
        return dict(case=case, batcher=table[0]["scene"], table=table)
    mesh, view = _scene(case["scene"], seed)
    if kind == "mesh":
        return dict(case=case, ctx=prt.Context(0), soup=_soup(case, mesh), names=["ground", "rock", "glass"])
    ctx = _context(mesh, case.get("high", True))
    state = dict(case=case, ctx=ctx)
    if kind in ("closest", "rebuild"):
        state.update(rays=_rays(case, mesh, seed),
                     hits=torch.empty((case["rays"], 4), dtype=torch.float32, device="cuda"))
    elif kind == "occluded":
        state.update(rays=_rays(case, mesh, seed), t=torch.empty(case["rays"], dtype=torch.float32, device="cuda"))
    else:
        w, h = case["width"], case["height"]
        ctx.init_frame(w, h)
        ctx.set_view(_view(case, view), w, h)
        state["accum"] = torch.empty((h, w, 4), dtype=torch.float32, device="cuda")
        if kind == "frame":
            ctx.set_integrator(case["integrator"])
            if case["albedo"]:
                ctx.set_albedo(torch.from_numpy(scenes.albedo_for(mesh, seed)).cuda())
            if case["packets"] or case["wave"]:
                paths = case["wave"] * ((w + 7) // 8) * ((h + 7) // 8) * 64
                ctx.set_tune(128, 0, paths, 2, case["packets"])
        elif kind == "train":
            albedo, target = _train_inputs(case, mesh, seed)
            state.update(albedo=albedo, target=target, d_albedo=torch.empty_like(albedo),
                         d_sky=torch.empty(1, dtype=torch.float32, device="cuda"))
    torch.cuda.synchronize()
    return state


# --- one pass ---------------------------------------------------------------

def _hits(hits):
    return {"t": hits[:, 0], "prim": hits.view(torch.int32)[:, 1], "u": hits[:, 2], "v": hits[:, 3]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        stats = state["batcher"].render_batch(state["table"])
        return {"rays": stats["ray"], "images": [q["accum"] for q in state["table"]]}
    ctx = state["ctx"]
    if kind == "closest":
        ctx.intersect(state["rays"], state["hits"], case["rays"])
        return _hits(state["hits"])
    if kind == "rebuild":
        ctx.build()
        ctx.intersect(state["rays"], state["hits"], case["rays"])
        return _hits(state["hits"])
    if kind == "occluded":
        ctx.occluded(state["rays"], state["t"], case["rays"])
        # which hit's distance comes back is left open by the call: an application uses whether there is one
        return state["t"] >= 0
    if kind == "frame":
        stats = ctx.render(case["spp"], case["depth"], accumulate=False)
        ctx.read_accum(state["accum"])
        return {"rays": stats["ray"], "image": state["accum"]}
    if kind == "viewer":
        stats = ctx.render(1, case["depth"], accumulate=True)
        ctx.read_accum(state["accum"])
        return {"rays": stats["ray"], "image": state["accum"]}
    if kind == "train":
        spp, accum = case["spp"], state["accum"]
        ctx.set_albedo(state["albedo"])
        ctx.set_sky(0.9)
        ctx.clear()
        ctx.render(spp, case["depth"], accumulate=True)
        ctx.read_accum(accum)
        # L = mean over pixels and channels of (accum / spp - target)^2
        d_sum = (accum[..., :3] / spp - state["target"]) * (2.0 / (state["target"].numel() * spp))
        torch.cuda.current_stream().synchronize()
        ctx.render_backward(0, spp, case["depth"], d_sum, state["d_albedo"], state["d_sky"])
        return {"image": accum, "d_albedo": state["d_albedo"], "d_sky": state["d_sky"]}
    ctx.build_mesh(state["soup"], state["names"])
    return {k: v for k, v in ctx.read_built_mesh().items() if v is not None}


# --- what a pass cannot do without --------------------------------------------

def work(case):
    kind = case["kind"]

    def ray_flops(scene, rays):
        # an 8-wide tree: per level 8 box tests of 6 multiply-adds and 6 min/max, then two triangle tests and a bounce
        levels = max(1.0, math.log(TRIANGLES[scene], 8))
        return rays * (levels * 8 * 18 + 2 * 60 + 100)

    if kind == "batch":
        reqs = _requests(case)
        pixels = sum(q["width"] * q["height"] for q in reqs)
        return {"bytes": 16 * pixels + 36 * sum(TRIANGLES[s] for s in {q["scene"] for q in reqs}),
                "flops": sum(ray_flops(q["scene"], 2 * q["width"] * q["height"] * q["spp"]) for q in reqs)}
    tris = TRIANGLES[case["scene"]]
    if kind == "mesh":
        # soup records in; indices, material ids and about half as many vertices out
        return {"bytes": (100 + 12 + 4 + 6 + (6 if case["normals"] else 0)) * tris, "flops": 9 * tris}
    if kind == "closest":
        return {"bytes": 48 * case["rays"], "flops": ray_flops(case["scene"], case["rays"])}
    if kind == "occluded":
        return {"bytes": 36 * case["rays"], "flops": ray_flops(case["scene"], case["rays"])}
    if kind == "rebuild":
        # index and vertex reads, the leaf triangles and about 0.2 nodes of 80 bytes per triangle written
        return {"bytes": 48 * case["rays"] + (12 + 6 + 48 + 16) * tris,
                "flops": ray_flops(case["scene"], case["rays"]) + 60.0 * tris * math.log2(tris)}
    pixels = case["width"] * case["height"]
    paths = pixels * case.get("spp", 1)
    if kind == "train":
        # the image, the target and the gradient image; albedo and its gradient; the paths twice
        return {"bytes": 40 * pixels + 44 * tris, "flops": 2 * ray_flops(case["scene"], 2 * paths)}
    rays = (3 if case.get("integrator") == "diffuse2" else 2) * paths
    return {"bytes": 16 * pixels + 36 * tris, "flops": ray_flops(case["scene"], rays)}


# --- the same results in 64 bits ----------------------------------------------

_GROUP = 128   # consecutive triangles that share a box in the search


class _Triangles64:
    def __init__(self, mesh):
        p = torch.from_numpy(mesh.positions).cuda().double()
        v = p[torch.from_numpy(mesh.indices).cuda().long()]                    # (T, 3, 3)
        self.n = len(v)
        pad = (-self.n) % _GROUP
        v = torch.cat([v, v[-1:].expand(pad, 3, 3)]) if pad else v
        g = v.reshape(-1, 3 * _GROUP, 3)
        self.lo, self.hi = g.amin(1) - 1e-9, g.amax(1) + 1e-9                  # (G, 3)
        self.v0, self.e1, self.e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]

    def closest(self, org, dir, tfar=math.inf):
        """t (inf: miss), triangle, u, v of the nearest hit in (0, tfar]."""
        n = len(org)
        t = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
        prim = torch.full((n,), -1, dtype=torch.int64, device="cuda")
        u, v = torch.zeros_like(t), torch.zeros_like(t)
        step = max(1, 40_000_000 // len(self.lo))
        for a in range(0, n, step):
            o, d = org[a:a + step], dir[a:a + step]
            near = torch.zeros((len(o), len(self.lo)), dtype=torch.float64, device="cuda")
            far = torch.full_like(near, tfar)
            for k in range(3):
                inv = 1.0 / torch.where(d[:, k].abs() > 1e-300, d[:, k], 1e-300)
                t0, t1 = (self.lo[:, k] - o[:, k:k + 1]) * inv[:, None], (self.hi[:, k] - o[:, k:k + 1]) * inv[:, None]
                near, far = torch.maximum(near, torch.minimum(t0, t1)), torch.minimum(far, torch.maximum(t0, t1))
            pairs = (near <= far * (1 + 1e-12)).nonzero()
            del near, far, t0, t1
            for b in range(0, len(pairs), 300_000):
                self._test(o, d, tfar, pairs[b:b + 300_000], a, t, prim, u, v)
        return t, prim, u, v

    def _test(self, o, d, tfar, pairs, at, t, prim, u, v):
        tri = (pairs[:, 1:] * _GROUP + torch.arange(_GROUP, device="cuda")).reshape(-1)
        ray = pairs[:, :1].expand(-1, _GROUP).reshape(-1)
        dd, e1, e2 = d[ray], self.e1[tri], self.e2[tri]
        p = torch.linalg.cross(dd, e2)
        inv = 1.0 / (e1 * p).sum(1)
        s = o[ray] - self.v0[tri]
        uu = (s * p).sum(1) * inv
        q = torch.linalg.cross(s, e1)
        vv = (dd * q).sum(1) * inv
        tt = (e2 * q).sum(1) * inv
        hit = ((uu >= 0) & (vv >= 0) & (uu + vv <= 1) & (tt > 0) & (tt <= tfar) & (tri < self.n)).nonzero()[:, 0]
        ray, tri, tt, uu, vv = ray[hit] + at, tri[hit], tt[hit], uu[hit], vv[hit]
        t.scatter_reduce_(0, ray, tt, "amin")
        best = (tt == t[ray]).nonzero()[:, 0]
        ray = ray[best]
        prim[ray], u[ray], v[ray] = tri[best], uu[best], vv[best]


_M32 = 0xFFFFFFFF


def _rotl(x, r):
    return ((x << r) | (x >> (32 - r))) & _M32


def _seed(pixel, sample):
    """Murmur3 of (pixel, pass), the state of the path's LCG."""
    h = torch.zeros_like(pixel)
    for k in (pixel, sample):
        k = _rotl((k * 0xCC9E2D51) & _M32, 15) * 0x1B873593 & _M32
        h = (_rotl(h ^ k, 13) * 5 + 0xE6546B64) & _M32
    h = ((h ^ (h >> 16)) * 0x85EBCA6B) & _M32
    h = ((h ^ (h >> 13)) * 0xC2B2AE35) & _M32
    return h ^ (h >> 16)


def _next(s):
    s = (s * 1664525 + 1013904223) & _M32
    return s, (s.float() * 2.0 ** -32).double()


def _unit(a):
    return a / a.norm(dim=1, keepdim=True)


def _camera_rays(cam, w, h, pixel, rng):
    f = {k: torch.tensor(list(getattr(cam, k)), dtype=torch.float64, device="cuda")
         for k in ("origin", "basisU", "basisV", "imageO", "imageDx", "imageDy")}
    rng, jx = _next(rng)
    rng, jy = _next(rng)
    rng, lx = _next(rng)
    rng, ly = _next(rng)
    d = (f["imageO"] + f["imageDx"] * (((pixel % w) + jx) / w)[:, None]
         + f["imageDy"] * (((pixel // w) + jy) / h)[:, None])
    if cam.lensRadius == 0:
        return rng, f["origin"].expand(len(pixel), 3), _unit(d)
    r, phi = lx.sqrt() * cam.lensRadius, 2 * math.pi * ly
    begin = f["origin"] + f["basisU"] * (r * phi.cos())[:, None] + f["basisV"] * (r * phi.sin())[:, None]
    return rng, begin, _unit(f["origin"] + d * cam.focalDistance - begin)


class _Frame64:
    """The shading frame at the hits of rays, and cosine-weighted rays leaving it."""

    def __init__(self, tris, org, dir, t, prim):
        self.p = org + t[:, None] * dir
        self.eps = torch.maximum(t, self.p.abs().amax(1)) * (float.fromhex("0x1.fp-18"))
        n = _unit(torch.linalg.cross(tris.e1[prim], tris.e2[prim]))
        self.n = torch.where(((n * dir).sum(1) > 0)[:, None], -n, n)
        x, y, z = self.n.unbind(1)
        zero = torch.zeros_like(x)
        u0, u1 = torch.stack([zero, z, -y], 1), torch.stack([-z, zero, x], 1)
        self.u = _unit(torch.where(((u0 * u0).sum(1) > (u1 * u1).sum(1))[:, None], u0, u1))
        self.v = _unit(torch.linalg.cross(self.n, self.u))

    def sample(self, rng):
        rng, sx = _next(rng)
        rng, sy = _next(rng)
        sin, phi = (1 - sx).sqrt(), 2 * math.pi * sy
        d = (self.u * (phi.cos() * sin)[:, None] + self.v * (phi.sin() * sin)[:, None] + self.n * sx.sqrt()[:, None])
        return rng, self.p + self.eps[:, None] * d, d


def _image64(mesh, cam, w, h, spp, depth, nee=False, albedo=None, sky=1.0, on_path=None):
    """The accumulated (h, w, 4) sums of passes 0..spp-1, one pass at a time;
    on_path(pixel, throughput, prims) sees the paths that escape."""
    tris = _Triangles64(mesh)
    image = torch.zeros((w * h, 4), dtype=torch.float64, device="cuda")
    alb = torch.full((mesh.tri_count,), 0.8, dtype=torch.float64, device="cuda") if albedo is None else albedo.double()
    for sample in range(spp):
        pixel = torch.arange(w * h, device="cuda")
        rng = _seed(pixel, torch.full_like(pixel, sample))
        rng, org, dir = _camera_rays(cam, w, h, pixel, rng)
        thr = torch.ones(w * h, dtype=torch.float64, device="cuda")
        prims = torch.full((w * h, 0), -1, dtype=torch.int64, device="cuda")
        for k in range(depth + 1):
            t, prim, _, _ = tris.closest(org, dir)
            out, hit = torch.isinf(t), ~torch.isinf(t)
            image[:, :3].index_add_(0, pixel[out], (thr[out] * sky * (0.5 if nee and k else 1.0))[:, None].expand(-1, 3))
            if on_path:
                on_path(pixel[out], thr[out], prims[out])
            if k == depth or not bool(hit.any()):
                break
            pixel, rng, prim, thr = pixel[hit], rng[hit], prim[hit], thr[hit] * alb[prim[hit]]
            prims = torch.cat([prims[hit], prim[:, None]], 1)
            frame = _Frame64(tris, org[hit], dir[hit], t[hit], prim)
            if nee:
                rng, so, sd = frame.sample(rng)
                free = torch.isinf(tris.closest(so, sd)[0])
                image[:, :3].index_add_(0, pixel[free], (thr[free] * sky * 0.5)[:, None].expand(-1, 3))
            rng, org, dir = frame.sample(rng)
        image[:, 3] += 1
    return image.reshape(h, w, 4)


def _heavy(case, rays):
    """Whether the search of so many rays would take over about 10 seconds."""
    groups = TRIANGLES[case["scene"]] / _GROUP
    return rays * (groups * 30 + 40000) > 3.0e12


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("closest", "rebuild", "frame", "viewer", "train"):
        return None   # whole numbers (occlusion flags, indexed meshes) or too much work (batches)
    paths = case["rays"] if "rays" in case else case["width"] * case["height"] * case.get("spp", 1)
    rays = paths * (1 if "rays" in case else 4.5 if case.get("integrator") == "diffuse2" else 2.5)
    if _heavy(case, rays):
        return None
    mesh, view = _scene(case["scene"], seed)
    if "rays" in case:
        r = _rays(case, mesh, seed).double()
        t, _, u, v = _Triangles64(mesh).closest(r[:, 0:3], r[:, 4:7])
        return {"t": torch.where(torch.isinf(t), -1.0, t), "prim": None, "u": u, "v": v}
    w, h, spp, depth = case["width"], case["height"], case.get("spp", 1), case["depth"]
    cam = prt.camera_from_view(_view(case, view), w, h)
    if kind != "train":
        albedo = torch.from_numpy(scenes.albedo_for(mesh, seed)).cuda() if case.get("albedo") else None
        nee = case.get("integrator") == "diffuse2"
        return {"rays": None, "image": _image64(mesh, cam, w, h, spp, depth, nee, albedo)}
    albedo, target = (x.double() for x in _train_inputs(case, mesh, seed))
    ends = []
    image = _image64(mesh, cam, w, h, spp, depth, albedo=albedo, sky=0.9, on_path=lambda *e: ends.append(e))
    g = ((image[..., :3] / spp - target) * (2.0 / (target.numel() * spp))).sum(-1).reshape(-1)
    d_albedo, d_sky = torch.zeros_like(albedo), torch.zeros(1, dtype=torch.float64, device="cuda")
    for pixel, thr, prims in ends:
        d_sky += (g[pixel] * thr).sum()
        for k in range(prims.shape[1]):
            d_albedo.index_add_(0, prims[:, k], g[pixel] * thr * 0.9 / albedo[prims[:, k]])
    return {"image": image, "d_albedo": d_albedo, "d_sky": d_sky}
