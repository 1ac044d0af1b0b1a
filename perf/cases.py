"""The workloads whose time this project is judged by, through its public entry points: `Scene`,
the integrators, the render service and the C ABI behind them.

Five kinds of work:

  trace   closest hits of a batch of rays (`Scene.intersection` on host arrays, `xtgpu_trace` on
          device buffers): camera rays, or rays that leave the surface those hit
  frame   one frame into host memory, as `Scene.render` and the integrator classes return it
  device  one frame into a device buffer (`xtgpu_render`)
  serve   a mix of jobs over eight resident scenes on the render service, frames read in host memory
  load    a scene uploaded, its trees built, and a first depth preview of it

Scenes come from the seeded generators of `xtracer_b200.scenes`; the seed of a state moves the geometry,
the rays and the sample streams, never the sizes.
"""
import ctypes
import math

import numpy as np
import torch

from xtracer_b200 import scenes, xtgpu
from xtracer_b200.service import Service

FORMATS = {"fp32": xtgpu.NODES_FP32, "q8": xtgpu.NODES_Q8, "w8": xtgpu.NODES_W8}
INTEGRATORS = {"stencil": xtgpu.STENCIL, "depth": xtgpu.DEPTH, "ao": xtgpu.AO, "path": xtgpu.PATHTRACER,
               "normal": xtgpu.NORMAL, "uv": xtgpu.UV, "emission": xtgpu.EMISSION, "wireframe": xtgpu.WIREFRAME}
CLASSES = {"depth": xtgpu.DepthIntegrator, "stencil": xtgpu.StencilIntegrator, "ao": xtgpu.AOIntegrator,
           "path": xtgpu.PathtracerIntegrator, "normal": xtgpu.NormalIntegrator, "uv": xtgpu.UVIntegrator,
           "emission": xtgpu.EmissionIntegrator, "wireframe": xtgpu.WireframeIntegrator}


def _render(name, kind, integrator, scene, size, width, height, spp, depth, fmt, leaf, aa=1, jitter=False,
            ao_distance=100.0, rect=""):
    c = {"kind": kind, "integrator": integrator, "scene": scene, "size": size, "width": width, "height": height,
         "spp": spp, "depth": depth, "format": fmt, "leaf": leaf, "aa": aa, "jitter": jitter,
         "ao_distance": ao_distance, "rect": rect}
    return dict(c, name=name) if name else c


def _trace(name, scene, size, rays, fmt, leaf, host, bounce):
    c = {"kind": "trace", "scene": scene, "size": size, "rays": rays, "format": fmt, "leaf": leaf, "host": host,
         "bounce": bounce}
    return dict(c, name=name) if name else c


def listed():
    return [
        # Picking and probing from host code: a thousand rays against a small scene.  Launches and copies.
        _trace("pick_spheres64", "spheres", 64, 1000, "fp32", 2, True, False),
        # A depth preview while a scene is set up, with the defaults of the integrator classes.
        _render("preview_depth_terrain10k", "frame", "depth", "terrain", 10000, 320, 240, 1, 1, "fp32", 2),
        # One region of a textured frame rendered again after an edit: a few tiles, bilinear textures, ERP sky.
        _render("region_path_textured", "frame", "path", "textured", 0, 640, 480, 16, 4, "fp32", 2,
                rect="288,200,352,264"),
        # The plain small pathtracer job: 64 spheres over a plane, 256 x 256, 16 spp, depth 4, host frame.
        _render("path_spheres64_256", "frame", "path", "spheres", 64, 256, 256, 16, 4, "fp32", 2),
        # Primary rays of a full-HD frame over the 1M-triangle terrain, default tree.
        _render("depth_terrain1m_1080p", "device", "depth", "terrain", 1000000, 1920, 1080, 1, 1, "fp32", 2),
        # Incoherent occlusion rays on the 2M-triangle hairball, the 8-wide tree.
        _render("ao_hairball2m_512", "device", "ao", "hairball", 2000000, 512, 512, 16, 1, "w8", 1,
                ao_distance=0.2),
        # Final-quality path tracing of a mesh, 8-wide tree, several bounces.
        _render("path_terrain200k_1024", "device", "path", "terrain", 200000, 1024, 1024, 4, 4, "w8", 1),
        # Phong and Blinn-Phong meshes with mesh and sphere lights, depth 8, an odd frame, quantised binary nodes.
        _render("path_phong_q8_odd", "device", "path", "phong", 160000, 641, 359, 8, 8, "q8", 2),
        # A wavefront of bounce rays traced for a caller's own integrator, device buffers.
        _trace("trace_bounce_hairball1m", "hairball", 1000000, 1 << 20, "w8", 1, False, True),
        # A ragged batch of camera rays on the default tree.
        _trace("trace_camera_terrain200k", "terrain", 200000, 77777, "fp32", 2, False, False),
        # The render service: uneven jobs over eight resident scenes, admitted together, three waves in flight.
        {"name": "serve_mix", "kind": "serve", "jobs": 24, "mix": 4, "scale": 0.1, "most": 512, "format": "w8"},
        # Opening a scene: upload, default and 8-wide trees, first preview.
        {"name": "load_terrain500k", "kind": "load", "scene": "terrain", "size": 500000, "leaf": 1, "formats": "fp32,w8"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _any_scene(rng):
    scene = rng.choice(["spheres", "terrain", "terrain", "hairball", "phong", "textured"])
    size = {"spheres": lambda: _log(rng, 8, 4096), "terrain": lambda: _log(rng, 1000, 500000),
            "hairball": lambda: _log(rng, 1000, 500000), "phong": lambda: _log(rng, 2000, 200000),
            "textured": lambda: 0}[scene]()
    return scene, size


def draw(rng):
    kind = rng.choice(["trace", "trace", "frame", "frame", "device", "device", "device", "serve", "load"])
    fmt, leaf = rng.choice(["fp32", "q8", "w8", "w8"]), rng.choice([1, 1, 2, 3])
    scene, size = _any_scene(rng)
    if kind == "trace":
        host = rng.random() < 0.4
        return _trace(None, scene, size, _log(rng, 100, 200000 if host else 1 << 20), fmt, leaf, host,
                      rng.random() < 0.5)
    if kind == "serve":
        return {"kind": "serve", "jobs": rng.randint(3, 32), "mix": rng.randint(1, 1 << 20),
                "scale": round(rng.uniform(0.02, 0.1), 3), "most": rng.choice([128, 256, 512]),
                "format": rng.choice(["fp32", "w8", "w8"])}
    if kind == "load":
        scene = rng.choice(["spheres", "terrain", "hairball"])
        size = _log(rng, 500, 4096) if scene == "spheres" else _log(rng, 2000, 500000)
        return {"kind": "load", "scene": scene, "size": size, "leaf": leaf,
                "formats": rng.choice(["fp32", "q8", "fp32,w8", "w8"])}
    integrator = rng.choice(["path", "path", "path", "ao", "ao", "depth", "depth", "stencil", "normal", "uv", "emission",
                             "wireframe"])
    most = 512 if kind == "frame" else 1280
    width, height = _log(rng, 33, most), _log(rng, 33, most)
    aa = rng.choice([1, 1, 1, 2, 3])
    jitter = rng.random() < 0.3
    per = aa if jitter else aa * aa
    spp = max(1, min(_log(rng, 1, 32), 4000000 // (width * height * per)))
    rect = ""
    if kind == "frame" and rng.random() < 0.3:
        x0, y0 = rng.randint(0, width - 33), rng.randint(0, height - 33)
        rect = "%d,%d,%d,%d" % (x0, y0, rng.randint(x0 + 33, width), rng.randint(y0 + 33, height))
    return _render(None, kind, integrator, scene, size, width, height, spp, rng.randint(1, 8), fmt, leaf, aa, jitter,
                   rng.choice([0.2, 5.0, 100.0]), rect)


# ---------------------------------------------------------------------------------------------------------------


def _spec(scene, size, seed):
    if scene == "spheres":
        return scenes.spheres_scene(size, seed=seed, extent=max(5.0, 0.625 * math.sqrt(size)))
    if scene == "terrain":
        return scenes.terrain_scene(size, seed=seed)
    if scene == "hairball":
        return scenes.hairball_scene(size, seed=seed)
    if scene == "phong":
        return scenes.precision_scene(size / 8.0e6, seed=seed % 100000)
    return scenes.textured_scene("erp", seed=seed)


def _basis(camera):
    """Camera position and axes in 64 bits; the horizontal field of view gives the depth of the image plane."""
    pos = np.array(camera.position, np.float64)
    z = np.array(camera.target, np.float64) - pos
    z /= np.linalg.norm(z)
    x = np.cross(np.array(camera.up, np.float64), z)
    x /= np.linalg.norm(x)
    y = np.cross(x, z)
    y /= np.linalg.norm(y)
    return pos, x, y, z, 1.0 / math.tan(camera.fov * 0.017453292519943 / 2.0)


def _camera_dirs(camera, px, py, width, height):
    """Directions through the image positions (px, py), 64-bit torch tensors."""
    _, x, y, z, dz = _basis(camera)
    x, y, z = (torch.from_numpy(v).to(px) for v in (x, y, z))
    dx, dy = 2.0 * px / width - 1.0, (2.0 * py / height - 1.0) * (height / width)
    d = dx[:, None] * x + dy[:, None] * y + dz * z
    return d / d.norm(dim=1, keepdim=True)


def _camera_rays(spec, n, seed):
    """n camera rays in raster order, each at a random place in its pixel: (n, 4) float32 tensors on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = int(math.ceil(math.sqrt(n)))
    i = torch.arange(n, device="cuda")
    u = torch.rand((n, 2), generator=g, device="cuda", dtype=torch.float64)
    d = _camera_dirs(spec.camera, (i % w) + u[:, 0], (i // w) + u[:, 1], w, w)
    org, dirs = torch.zeros((n, 4), device="cuda"), torch.empty((n, 4), device="cuda")
    org[:, :3] = torch.tensor(spec.camera.position, device="cuda")
    dirs[:, :3], dirs[:, 3] = d.float(), math.inf
    return org, dirs


def _bounce_rays(spec, sc, fmt, org, dirs, seed):
    """The rays one bounce on: from each hit point, cosine-distributed about the normal that faces the ray.
    Rays that met nothing stay as they are."""
    n = org.shape[0]
    hits = torch.empty((n, 4), device="cuda")
    xtgpu.check(xtgpu.lib().xtgpu_trace(sc.handle, n, org.data_ptr(), dirs.data_ptr(), hits.data_ptr(), fmt, None))
    prim = hits.view(torch.int32)[:, 1].long()
    nt, ns = spec.n_tris, spec.spheres.shape[0]
    hit = prim >= 0
    p = org[:, :3].double() + dirs[:, :3].double() * torch.where(hit, hits[:, 0], torch.zeros(())).double()[:, None]
    nrm = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    is_t, is_s, is_p = hit & (prim < nt), (prim >= nt) & (prim < nt + ns), prim >= nt + ns
    if nt:
        v = torch.from_numpy(spec.tris).cuda()[prim[is_t]].double()
        nrm[is_t] = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    if ns:
        nrm[is_s] = p[is_s] - torch.from_numpy(spec.spheres).cuda()[prim[is_s] - nt, :3].double()
    if len(spec.planes):
        nrm[is_p] = torch.from_numpy(spec.planes).cuda()[prim[is_p] - nt - ns, :3].double()
    nrm /= nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
    nrm *= -torch.sign((nrm * dirs[:, :3].double()).sum(1, keepdim=True))
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    s = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    s = nrm + s / s.norm(dim=1, keepdim=True)
    s /= s.norm(dim=1, keepdim=True).clamp_min(1e-12)
    o2, d2 = org.clone(), dirs.clone()
    far = p.abs().amax(1, keepdim=True)
    o2[:, :3] = torch.where(hit[:, None], p + nrm * 1e-4 * (1.0 + far), org[:, :3].double()).float()
    d2[:, :3] = torch.where(hit[:, None], s, dirs[:, :3].double()).float()
    return o2, d2


def _formats(fmt):
    # the 8-wide tree is served beside the default one, which camera rays take
    return (xtgpu.NODES_FP32, xtgpu.NODES_W8) if fmt == "w8" else (FORMATS[fmt],)


SERVED = [("terrain", 10000), ("terrain", 50000), ("terrain", 200000), ("terrain", 500000), ("terrain", 1000000),
          ("hairball", 2000000), ("spheres", 64), ("spheres", 4096)]


def _served_jobs(case):
    """(scene, resolution, spp) of each job: every run of a case has the same ones."""
    rng = np.random.default_rng(case["mix"])
    sizes = [r for r in (128, 256, 512) if r <= case["most"]]
    return [(int(rng.integers(0, len(SERVED))), int(rng.choice(sizes)), int(rng.choice((1, 4, 16))))
            for _ in range(case["jobs"])]


def _rect(case):
    return tuple(int(v) for v in case["rect"].split(",")) if case["rect"] else None


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        specs = [_spec(s, n if s == "spheres" else max(8, int(n * case["scale"])), seed + k)
                 for k, (s, n) in enumerate(SERVED)]
        resident = [xtgpu.Scene(s, node_formats=_formats(case["format"]), leaf_size=1) for s in specs]
        svc = Service(resident, node_format=FORMATS[case["format"]], host_results=True, waves_in_flight=3)
        frames = [np.zeros((r, r, 4), np.float32) for _, r, _ in _served_jobs(case)]
        return {"case": case, "seed": seed, "scenes": resident, "service": svc, "frames": frames}
    spec = _spec(case["scene"], case["size"], seed)
    if kind == "load":
        fmts = tuple(FORMATS[f] for f in case["formats"].split(","))
        return {"case": case, "spec": spec, "formats": fmts}
    fmt = FORMATS[case["format"]]
    sc = xtgpu.Scene(spec, node_formats=_formats(case["format"]), leaf_size=case["leaf"])
    state = {"case": case, "seed": seed, "scene": sc, "format": fmt}
    if kind == "trace":
        org, dirs = _camera_rays(spec, case["rays"], seed)
        if case["bounce"]:
            org, dirs = _bounce_rays(spec, sc, fmt, org, dirs, seed)
        if case["host"]:
            state.update(org=org[:, :3].cpu().numpy().copy(), dirs=dirs[:, :3].cpu().numpy().copy())
        else:
            state.update(org=org, dirs=dirs, hits=torch.empty((case["rays"], 4), device="cuda"))
        return state
    dist = xtgpu.SAMPLES_RANDOM if case["jitter"] else xtgpu.SAMPLES_GRID
    if kind == "frame":
        p = xtgpu.Params(case["width"], case["height"], case["spp"], case["depth"], seed, fmt, case["ao_distance"],
                         case["aa"], dist)
        state["integrator"] = CLASSES[case["integrator"]]()
        state["integrator"].setup(xtgpu.Context(sc, p))
        return state
    state["params"] = xtgpu.RenderParams(INTEGRATORS[case["integrator"]], case["width"], case["height"], case["spp"],
                                         case["depth"], case["ao_distance"], seed, fmt, 0, 0, 0, 0, case["aa"], dist)
    state["frame"] = torch.empty((case["height"], case["width"], 4), device="cuda")
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "trace":
        sc, fmt = state["scene"], state["format"]
        if case["host"]:
            h = sc.intersection(state["org"], state["dirs"], node_format=fmt)
            return {"t": h["t"], "prim": h["prim"].view(np.int32), "u": h["u"], "v": h["v"]}
        hits = state["hits"]
        xtgpu.check(xtgpu.lib().xtgpu_trace(sc.handle, case["rays"], state["org"].data_ptr(), state["dirs"].data_ptr(),
                                            hits.data_ptr(), fmt, None))
        return {"t": hits[:, 0], "prim": hits.view(torch.int32)[:, 1], "u": hits[:, 2], "v": hits[:, 3]}
    if kind == "frame":
        if not case["rect"]:
            return state["integrator"].render()
        p = state["integrator"].ctx.params
        img, _ = state["scene"].render(INTEGRATORS[case["integrator"]], p.width, p.height, p.samples, p.rdepth,
                                       p.ao_max_distance, p.seed, p.node_format, _rect(case), p.aa,
                                       p.sample_distribution)
        return img
    if kind == "device":
        rays = ctypes.c_uint64()
        xtgpu.check(xtgpu.lib().xtgpu_render(state["scene"].handle, ctypes.byref(state["params"]),
                                             state["frame"].data_ptr(), ctypes.byref(rays), None))
        return {"frame": state["frame"], "rays": int(rays.value)}
    if kind == "serve":
        svc = state["service"]
        jobs = [svc.submit(s, xtgpu.PATHTRACER, r, r, spp, 4, seed=state["seed"] * 1000 + k)
                for k, (s, r, spp) in enumerate(_served_jobs(case))]
        svc.run()
        for jid, frame in zip(jobs, state["frames"]):
            svc.result(jid, frame)
            svc.release(jid)
        return state["frames"]
    sc = xtgpu.Scene(state["spec"], node_formats=state["formats"], leaf_size=case["leaf"])
    img, _ = sc.render(xtgpu.DEPTH, 320, 180, node_format=state["formats"][-1])
    sc.close()
    return img


# ---------------------------------------------------------------------------------------------------------------


def _prims(scene, size):
    return {"spheres": size + 2, "textured": 260}.get(scene, size)


def _ray_flops(prims):
    # a path from the root to one leaf, both children's boxes at each level, and two primitives
    return 48.0 * math.log2(prims + 1) + 120.0


def _path_rays(integrator, depth):
    # a camera ray; AO and the pathtracer go on from what it hits
    return 2 if integrator == "ao" or (integrator == "path" and depth > 1) else 1


def work(case):
    kind = case["kind"]
    if kind == "serve":
        b = f = 0.0
        for s, n in SERVED:
            b += 48.0 * (n if s == "spheres" else n * case["scale"])
        for s, r, spp in _served_jobs(case):
            b += 16.0 * r * r
            f += 2.0 * r * r * spp * _ray_flops(SERVED[s][1] if SERVED[s][0] == "spheres" else
                                                SERVED[s][1] * case["scale"] + 8)
        return {"bytes": b, "flops": f}
    prims = _prims(case["scene"], case["size"])
    if kind == "load":
        # the corners in, leaf primitives and nodes out; codes, sort passes and boxes
        out = 48.0 + sum({"fp32": 64.0, "q8": 32.0, "w8": 65.0}[x] for x in case["formats"].split(","))
        return {"bytes": prims * (36.0 + out) + 16.0 * 320 * 180, "flops": 150.0 * prims}
    if kind == "trace":
        return {"bytes": 48.0 * prims + 48.0 * case["rays"], "flops": case["rays"] * _ray_flops(prims)}
    x0, y0, x1, y1 = _rect(case) or (0, 0, case["width"], case["height"])
    pix = (x1 - x0) * (y1 - y0)
    paths = pix * case["spp"] * (case["aa"] if case["jitter"] else case["aa"] ** 2)
    return {"bytes": 48.0 * prims + 16.0 * pix,
            "flops": float(paths) * _path_rays(case["integrator"], case["depth"]) * _ray_flops(prims)}


def _closest(spec, org, dirs):
    """Closest hits by testing every primitive in 64 bits: distance, primitive, barycentrics of a triangle."""
    n = org.shape[0]
    t = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    prim = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    bu, bv = torch.zeros_like(t), torch.zeros_like(t)
    nt, ns = spec.n_tris, spec.spheres.shape[0]

    def take(tt, first, u=None, v=None):
        best, k = tt.min(dim=1)
        near = best < t
        t[near], prim[near] = best[near], first + k[near]
        for b, x in ((bu, u), (bv, v)):
            b[near] = x[near, k[near]] if x is not None else 0.0

    miss = torch.full((), math.inf, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 24) // n)
    tris = torch.from_numpy(spec.tris).cuda().double()
    for a in range(0, nt, step):
        v0, e1, e2 = tris[a:a + step, 0], tris[a:a + step, 1] - tris[a:a + step, 0], tris[a:a + step, 2] - tris[a:a + step, 0]
        nrm = torch.linalg.cross(e1, e2)
        # (o - v0) x d gives both barycentrics, their signs by the determinant -d.n
        det = -(dirs @ nrm.T)
        f = org[:, None] - v0[None]
        q = torch.linalg.cross(f, dirs[:, None].expand_as(f), dim=2)
        u, v = (q * e2).sum(2) / det, -(q * e1).sum(2) / det
        tt = (f * nrm).sum(2) / det
        ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (tt > 0)
        take(torch.where(ok, tt, miss), a, u, v)
    sph = torch.from_numpy(spec.spheres).cuda().double()
    for a in range(0, ns, step):
        f = org[:, None] - sph[None, a:a + step, :3]
        b, c = (f * dirs[:, None]).sum(2), (f * f).sum(2) - sph[None, a:a + step, 3] ** 2
        dd = (dirs * dirs).sum(1)[:, None]
        disc = b * b - dd * c
        tt = (-b - disc.clamp_min(0).sqrt()) / dd
        take(torch.where((disc > 0) & (tt > 0), tt, miss), nt + a)
    if len(spec.planes):
        pl = torch.from_numpy(spec.planes).cuda().double()
        nd = dirs @ pl[:, :3].T
        p0 = pl[:, :3].abs() * pl[:, 3:]
        tt = ((p0[None] - org[:, None]) * pl[None, :, :3]).sum(2) / nd
        take(torch.where((nd.abs() >= 1e-8) & (tt > 0), tt, miss), nt + ns)
    return t, prim, bu, bv


def exact(case, seed):
    """Distances and depth frames of scenes small enough for every primitive to be tested in 64 bits.  Which of two
    primitives at one distance is named, and AO and path-traced frames, which are sums over random samples, have no
    such value."""
    if case["kind"] == "trace":
        if case["bounce"] or case["rays"] * _prims(case["scene"], case["size"]) > 2e9:
            return None
        spec = _spec(case["scene"], case["size"], seed)
        org, dirs = _camera_rays(spec, case["rays"], seed)
        t, _, u, v = _closest(spec, org[:, :3].double(), dirs[:, :3].double())
        return {"t": t, "prim": None, "u": u, "v": v}
    if case["kind"] not in ("frame", "device") or case["integrator"] not in ("depth", "stencil") or case["rect"] or \
            case["jitter"] or case["aa"] != 1:
        return None
    w, h = case["width"], case["height"]
    if w * h * _prims(case["scene"], case["size"]) > 2e9:
        return None
    spec = _spec(case["scene"], case["size"], seed)
    i = torch.arange(w * h, device="cuda")
    dirs = _camera_dirs(spec.camera, (i % w).double() + 0.5, (i // w).double() + 0.5, w, h)
    org = torch.tensor(spec.camera.position, dtype=torch.float64, device="cuda").expand(w * h, 3)
    t, _, _, _ = _closest(spec, org, dirs)
    hit = torch.isfinite(t)
    img = torch.zeros((w * h, 4), dtype=torch.float64, device="cuda")
    if case["integrator"] == "stencil":
        img[hit] = 1.0
    else:
        img[:, :3] = torch.where(hit, (1.0 / torch.log(t)).clamp_min(0.0), torch.zeros_like(t))[:, None]
        img[:, 3] = 1.0
    img = img.reshape(h, w, 4)
    return img if case["kind"] == "frame" else {"frame": img, "rays": None}
