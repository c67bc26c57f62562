"""The work that a user of this framework has it do, as cases to be timed.

A case is one pass through the public entry points of cwbvh_b200:

  bake       AO rays of a surfel cache, traced any-hit, reduced to AO per
             surfel: the reference's main() flow (GenerateAORaysUniform,
             rtTrace, the reduction over a texel's rays)
  closest    closest hits of rays the caller already holds
  frame      camera rays, closest hits, surfels at the hits, one AO ray per
             hit, AO: a renderer's frame (the city configuration)
  batch      many resident scenes with their own rays in one launch
  instanced  camera rays through a two-level scene
  sort       Morton order of a ray buffer
  build      a mesh admitted on the device (GPU build) and baked at once
  serve      AO bake requests through the continuous-batching server, host
             surfels in and host AO out

Scenes are the repository's procedural ones (heightfield with boxes, city,
spheres over terrain); scene and rays come from the seed.  Any-hit passes
return the AO of every surfel, because which of a ray's occluders is reported
is not defined; closest passes return t and what belongs to the hit.
"""
import math

import numpy as np
import torch

import cwbvh_b200 as rq
from cwbvh_b200 import workloads as W

SPP = 32  # rays per texel of the reference's bake


def listed():
    return [
        # The smallest request that the serving workload sends: 4,096 rays.
        # A lightmap tile, an editor's preview: latency and launches count.
        dict(name="bake_4k", path="bake", scene="heightfield", tris=10592, kind="cwbvh", surfels=128, spp=SPP,
             fused=False),
        # The plain configuration: the 10,592-triangle scene with 1M AO rays.
        dict(name="bake_1m", path="bake", scene="heightfield", tris=10592, kind="cwbvh", surfels=32768, spp=SPP,
             fused=False),
        # The large configuration's scene family and its 4 rays per surfel,
        # past L2, an odd surfel count, counts kept instead of hits.
        dict(name="bake_spheres_16m", path="bake", scene="spheres", tris=8000000, kind="cwbvh", surfels=4000037, spp=4,
             fused=True),
        # The binary BVH on the small scene, ragged.
        dict(name="bake_bvh2", path="bake", scene="heightfield", tris=10592, kind="bvh2", surfels=26999, spp=37,
             fused=False),
        # Closest hits of incoherent rays: bounce rays, visibility with distance.
        dict(name="closest_1m", path="closest", scene="heightfield", tris=20000, kind="cwbvh", rays=1048576),
        # The binary BVH's closest hit, the reference's second kernel; odd count.
        dict(name="closest_bvh2", path="closest", scene="heightfield", tris=10592, kind="bvh2", rays=300007),
        # The city configuration: primary rays in 4x8-pixel tiles and AO from their hits.
        dict(name="frame_city", path="frame", scene="city", tris=937000, width=2048, height=2048),
        # The batched configuration's family: scenes of different sizes, each with its own rays.
        dict(name="batch_mixed", path="batch", scenes=12, tris_lo=10000, tris_hi=200000, surfels_lo=8192,
             surfels_hi=262144, spp=SPP),
        # Instances of city blocks under a top-level tree: primary rays.
        dict(name="instanced_city", path="instanced", instances=625, blocks=64, width=2048, height=2048),
        # Morton order of an incoherent ray buffer.
        dict(name="sort_4m", path="sort", scene="heightfield", tris=10592, rays=4194304),
        # A scene that must be ready at once: built on the device, then baked.
        dict(name="build_500k", path="build", scene="heightfield", tris=500000, surfels=32768, spp=SPP),
        # Bake requests of different sizes served together, host to host.
        dict(name="serve_bakes", path="serve", scenes=4, tris=10592, requests=24, surfels_lo=128, surfels_hi=32768,
             spp=SPP),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["bake", "bake", "bake", "closest", "closest", "frame", "batch", "instanced", "sort", "build",
                       "serve"])
    if path == "bake":
        scene = rng.choice(["heightfield", "city", "spheres"])
        kind = rng.choice(["cwbvh", "cwbvh", "bvh2"]) if scene == "heightfield" else "cwbvh"
        tris = _log(rng, 2000, 60000 if kind == "bvh2" else 200000) if scene == "heightfield" else \
            _log(rng, 20000, 900000) if scene == "city" else _log(rng, 50000, 4000000)
        spp = rng.choice([1, 4, 16, SPP, 37, 64])
        return dict(path=path, scene=scene, tris=tris, kind=kind, surfels=max(1, _log(rng, 4096, 8000000) // spp),
                    spp=spp, fused=rng.random() < 0.4)
    if path == "closest":
        kind = rng.choice(["cwbvh", "cwbvh", "bvh2"])
        return dict(path=path, scene="heightfield", tris=_log(rng, 2000, 60000 if kind == "bvh2" else 200000),
                    kind=kind, rays=_log(rng, 4096, 4000000))
    if path == "frame":
        return dict(path=path, scene="city", tris=_log(rng, 20000, 900000), width=4 * rng.randint(64, 500),
                    height=8 * rng.randint(32, 250))
    if path == "batch":
        return dict(path=path, scenes=rng.randint(2, 12), tris_lo=5000, tris_hi=_log(rng, 10000, 150000),
                    surfels_lo=128, surfels_hi=_log(rng, 1024, 200000), spp=rng.choice([8, SPP]))
    if path == "instanced":
        return dict(path=path, instances=rng.randint(16, 600), blocks=rng.randint(4, 64),
                    width=4 * rng.randint(64, 500), height=8 * rng.randint(32, 250))
    if path == "sort":
        return dict(path=path, scene="heightfield", tris=10592, rays=_log(rng, 4096, 4000000))
    if path == "build":
        return dict(path=path, scene=rng.choice(["heightfield", "city", "spheres"]), tris=_log(rng, 5000, 450000),
                    surfels=_log(rng, 256, 32768), spp=rng.choice([4, SPP]))
    return dict(path=path, scenes=rng.randint(1, 6), tris=_log(rng, 5000, 30000), requests=rng.randint(1, 24),
                surfels_lo=128, surfels_hi=_log(rng, 512, 32768), spp=rng.choice([16, SPP]))


# ------------------------------------------------------------------ scenes --

def _mesh(family, tris, seed):
    if family == "heightfield":
        return W.scene_of_size(seed, tris)
    if family == "city":
        return rq.gen_city(seed, max(1, tris // 94))
    return rq.gen_spheres_terrain(seed, tris)


def _scene(case, seed):
    """The scene with its mesh on the GPU.  Meshes past a million triangles
    are built on the device, the others by the host builder."""
    V, I = _mesh(case["scene"], case["tris"], seed)
    kind = rq.BVH2 if case.get("kind") == "bvh2" else rq.CWBVH
    if I.shape[0] > 1000000:
        v, i = torch.from_numpy(V).cuda(), torch.from_numpy(I).cuda()
        return W.DeviceScene(kind, None, rq.Scene.build_gpu(v, i), v, i, W.diag(V), I.shape[0])
    return W.upload(V, I, kind)


def _closest_views(hits):
    """t, u, v of a hit buffer.  The Woop address is left out: a triangle that
    the builder split has several, and which one is reported is not defined
    (2e-5 of the rays change it from run to run)."""
    return {"t": hits[:, 0], "u": hits[:, 2], "v": hits[:, 3]}


def _camera(lo, hi):
    ext = hi - lo
    eye = (float(lo[0] - 0.05 * ext[0]), float(lo[1] - 0.05 * ext[1]), float(0.25 * max(ext[0], ext[1])))
    look = (float(0.5 * (lo[0] + hi[0])), float(0.5 * (lo[1] + hi[1])), 0.0)
    return eye, look


def _sizes(stream, lo, hi, n):
    """The case's own sizes, the same for every seed."""
    return W.log_uniform(np.random.default_rng(stream), lo, hi, n).astype(np.int64)


# ----------------------------------------------------------------- prepare --

def prepare(case, seed):
    s = dict(case=case, seed=seed, ctx=rq.Context())
    path = case["path"]
    if path in ("bake", "closest", "sort"):
        ds = s["ds"] = _scene(case, seed)
    if path == "bake":
        n = case["surfels"] * case["spp"]
        s["pos"], s["nrm"], s["rad"] = rq.sample_surfels(ds.vertices, ds.indices, case["surfels"], seed + 1)
        s["rays"] = torch.empty((n, 8), device="cuda")
        s["hits"] = None if case["fused"] else torch.empty((n, 4), device="cuda")
    elif path == "closest":
        s["rays"] = W.ao_rays(ds, case["rays"], seed + 1)
        s["hits"] = torch.empty((case["rays"], 4), device="cuda")
        s["out"] = _closest_views(s["hits"])
    elif path == "sort":
        s["rays"] = W.ao_rays(ds, case["rays"], seed + 1)
        s["lo"], s["hi"] = ds.host.info["bounds_lo"], ds.host.info["bounds_hi"]
    elif path == "frame":
        V, I = _mesh("city", case["tris"], seed)
        s["scene"], s["diag"] = rq.Scene.from_host(rq.HostBVH(V, I)), W.diag(V)
        s["eye"], s["look"] = _camera(V.min(0), V.max(0))
        s["hits"] = torch.empty((case["width"] * case["height"], 4), device="cuda")
        s["ao_hits"] = torch.empty_like(s["hits"])
    elif path == "batch":
        tris = _sizes(1, case["tris_lo"], case["tris_hi"], case["scenes"])
        surfels = _sizes(2, case["surfels_lo"], case["surfels_hi"], case["scenes"])
        s["surfels"] = int(surfels.sum())
        s["hits"] = torch.empty((s["surfels"] * case["spp"], 4), device="cuda")
        items, at = [], 0
        for k, (t, m) in enumerate(zip(tris, surfels)):
            ds = W.upload(*W.scene_of_size(1000 * seed + k, int(t)))
            n = int(m) * case["spp"]
            items.append((ds.scene, W.ao_rays(ds, n, seed + k, spp=case["spp"]), s["hits"][at:at + n]))
            at += n
        s["batch"] = rq.Batch(s["ctx"], items, rq.ANY)
    elif path == "instanced":
        _prepare_instanced(s, case, seed)
    elif path == "build":
        V, I = _mesh(case["scene"], case["tris"], seed)
        s["v"], s["i"], s["diag"] = torch.from_numpy(V).cuda(), torch.from_numpy(I).cuda(), W.diag(V)
        n = case["surfels"] * case["spp"]
        s["pos"], s["nrm"], s["rad"] = rq.sample_surfels(s["v"], s["i"], case["surfels"], seed + 1)
        s["rays"], s["hits"] = torch.empty((n, 8), device="cuda"), torch.empty((n, 4), device="cuda")
    else:
        surfels = _sizes(2, case["surfels_lo"], case["surfels_hi"], case["requests"])
        s["server"] = rq.Server(hbm_budget_bytes=2 << 30, query=rq.ANY)
        s["requests"] = []
        scenes = [W.upload(*W.scene_of_size(1000 * seed + k, case["tris"])) for k in range(case["scenes"])]
        ids = [s["server"].add_scene(ds.scene) for ds in scenes]
        for k, m in enumerate(surfels):
            ds = scenes[k % len(scenes)]
            host = [torch.empty(x.shape, pin_memory=True).copy_(x).numpy()
                    for x in rq.sample_surfels(ds.vertices, ds.indices, int(m), seed + k)]
            ao = torch.empty(int(m), pin_memory=True).numpy()
            s["requests"].append((ids[k % len(ids)], host, ds.diag, seed + 77 + k, ao))
        torch.cuda.synchronize()
    return s


def _prepare_instanced(s, case, seed):
    """City blocks on a square grid of lots with quarter turns."""
    rng = np.random.default_rng(seed)
    meshes = [rq.gen_city(1000 * seed + k, 16) for k in range(case["blocks"])]
    s["blas"] = [rq.Scene.from_host(rq.HostBVH(V, I)) for V, I in meshes]
    n, lot = case["instances"], 80.0
    side = math.ceil(math.sqrt(n))
    which = rng.integers(0, len(meshes), n).astype(np.int32)
    turn = rng.integers(0, 4, n)
    M = np.zeros((n, 3, 4), np.float32)
    for k in range(n):
        c, t = [(1, 0), (0, 1), (-1, 0), (0, -1)][turn[k]]
        R = np.array([[c, -t, 0], [t, c, 0], [0, 0, 1]], np.float64)
        mid = np.array([lot / 2, lot / 2, 0.0])
        M[k, :, :3] = R
        M[k, :, 3] = np.array([(k % side) * lot, (k // side) * lot, 0.0]) + mid - R @ mid
    s["tlas"] = rq.Tlas(s["blas"], M, which)
    lo, hi = np.zeros(3), np.array([side * lot, math.ceil(n / side) * lot, 200.0])
    eye, look = _camera(lo, hi)
    w, h = case["width"], case["height"]
    far = 10.0 * float(np.linalg.norm(hi - lo))
    s["rays"] = rq.camera_rays(eye, look, (0.0, 0.0, 1.0), 60.0, w, h, 0.0, far, tile=(4, 8))
    s["hits"] = torch.empty((w * h, 4), device="cuda")
    s["inst"] = torch.empty(w * h, dtype=torch.int32, device="cuda")
    s["out"] = dict(_closest_views(s["hits"]), instance=s["inst"])


# --------------------------------------------------------------------- run --

def _bake(s, scene, diag):
    c = s["case"]
    rq.aorays(s["pos"], s["nrm"], s["rad"], c["spp"], s["seed"], 1e-4 * diag, 0.1 * diag, 0.0, out=s["rays"])
    if c.get("fused"):
        return {"occluded": rq.trace_ao(s["ctx"], scene, s["rays"], c["spp"])}
    rq.trace(s["ctx"], scene, s["rays"], s["hits"], rq.ANY)
    return {"ao": rq.ao_reduce(s["hits"], c["surfels"], c["spp"])}


def run(s):
    c = s["case"]
    path = c["path"]
    if path == "bake":
        return _bake(s, s["ds"].scene, s["ds"].diag)
    if path == "closest":
        rq.trace(s["ctx"], s["ds"].scene, s["rays"], s["hits"], rq.CLOSEST)
        return s["out"]
    if path == "frame":
        d = s["diag"]
        rays = rq.camera_rays(s["eye"], s["look"], (0.0, 0.0, 1.0), 60.0, c["width"], c["height"], 0.0, 10.0 * d,
                              tile=(4, 8))
        rq.trace(s["ctx"], s["scene"], rays, s["hits"], rq.CLOSEST)
        pos, nrm, rad = rq.surfels_from_hits(rays, s["hits"], s["scene"])
        ao_rays = rq.aorays(pos, nrm, rad, 1, s["seed"], 1e-4 * d, 0.05 * d, 0.0)
        rq.trace(s["ctx"], s["scene"], ao_rays, s["ao_hits"], rq.ANY)
        return {"t": s["hits"][:, 0], "pos": pos, "ao": rq.ao_reduce(s["ao_hits"], rays.shape[0], 1)}
    if path == "batch":
        s["batch"].run()
        return {"ao": rq.ao_reduce(s["hits"], s["surfels"], c["spp"])}
    if path == "instanced":
        rq.trace_instanced(s["ctx"], s["tlas"], s["rays"], s["hits"], rq.CLOSEST, instance_out=s["inst"])
        return s["out"]
    if path == "sort":
        rays, perm = rq.sort_rays(s["ctx"], s["rays"], s["lo"], s["hi"])
        return {"rays": rays, "perm": perm}
    if path == "build":
        s["scene"] = rq.Scene.build_gpu(s["v"], s["i"])
        return _bake(s, s["scene"], s["diag"])
    tickets = [s["server"].submit_bake(i, *host, c["spp"], seed, 1e-4 * d, 0.1 * d, 0.0, ao)
               for i, host, d, seed, ao in s["requests"]]
    for t in tickets:
        s["server"].wait(t)
    return [ao for _, _, _, _, ao in s["requests"]]


# -------------------------------------------------------------------- work --

def _rays(c):
    if c["path"] in ("bake", "build"):
        return c["surfels"] * c["spp"]
    if c["path"] in ("frame", "instanced"):
        return c["width"] * c["height"] * (2 if c["path"] == "frame" else 1)
    if c["path"] in ("batch", "serve"):
        n = c["scenes"] if c["path"] == "batch" else c["requests"]
        return int(_sizes(2, c["surfels_lo"], c["surfels_hi"], n).sum()) * c["spp"]
    return c["rays"]


def work(case):
    """Bytes: each input read and each output written once, the scene's
    triangles (48 B each) and nodes (80 B per 2.6 triangles) among the inputs.
    Operations: about 8 node tests of 48 multiply-adds and 3 triangle tests
    of 18 per ray; clustering and treelets are left out of a build's."""
    n, path = _rays(case), case["path"]
    flops = 0 if path == "sort" else n * (8 * 96 + 3 * 36)
    if path in ("batch", "serve"):
        tris = case["scenes"] * case["tris"] if path == "serve" else \
            int(_sizes(1, case["tris_lo"], case["tris_hi"], case["scenes"]).sum())
    else:
        tris = case["instances"] * 24 if path == "instanced" else 0 if path == "sort" else case["tris"]
    scene = tris * (48 + 80 / 2.6)
    if path == "bake":
        b = case["surfels"] * (36 + 4)
    elif path == "build":
        b = case["surfels"] * (36 + 4) + tris * 18
    elif path == "frame":
        b = n / 2 * (4 + 16 + 4)
    elif path == "serve":
        b = n / case["spp"] * (36 + 4)
    elif path == "batch":
        b = n * 32 + n / case["spp"] * 4
    elif path == "sort":
        b = n * (32 + 32 + 4)
    else:
        b = n * (32 + 16 + (4 if path == "instanced" else 0))
    return {"bytes": b + scene, "flops": flops}


# ------------------------------------------------------------------- exact --

_TESTS = 2.5e10  # ray-triangle pairs of an exhaustive test in 64 bits


def _philox(counter, seed):
    """Philox4x32-10 (Salmon et al., SC 2011), counter words (low, high, 0, 0)."""
    c = [counter & 0xFFFFFFFF, counter >> 32, torch.zeros_like(counter), torch.zeros_like(counter)]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF

    def mul(m, x):  # 32 x 32 -> (high, low) without leaving 63 bits
        lo, hi = (x & 0xFFFF) * m, (x >> 16) * m
        t = (lo >> 16) + (hi & 0xFFFFFFFF)
        return ((hi >> 32) << 16) + (t >> 16) & 0xFFFFFFFF, (x * m) & 0xFFFFFFFF

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _aorays64(pos, nrm, spp, seed):
    """Origins and directions of the AO rays in 64 bits (offset 0)."""
    n = pos.shape[0] * spp
    p, z = pos[:, :3].double(), nrm[:, :3].double()
    x = torch.linalg.cross(z, z.new_tensor([[0.0, 0.0, 1.0]]).expand_as(z))
    y = torch.linalg.cross(z, z.new_tensor([[0.0, 1.0, 0.0]]).expand_as(z))
    t1 = torch.where(x.norm(dim=1, keepdim=True) < 0.1, y, x)
    t1 = t1 / t1.norm(dim=1, keepdim=True)
    t2 = torch.linalg.cross(t1, z)
    t2 = t2 / t2.norm(dim=1, keepdim=True)
    r = _philox(torch.arange(n, dtype=torch.int64, device=pos.device), seed)
    a, b = ((2.0 * ((w >> 8) + 1).double() / 2 ** 24 - 1.0) for w in r[:2])
    wide = a * a > b * b
    rr = torch.where(wide, a, b)
    th = torch.where(wide, (math.pi / 4) * (b / a), math.pi / 2 - (math.pi / 4) * (a / b))
    th = torch.where((a == 0) & (b == 0), torch.zeros_like(th), th)
    u, v = rr * torch.cos(th), rr * torch.sin(th)
    w = torch.sqrt(torch.clamp(1.0 - u * u - v * v, min=0.0))
    rep = lambda q: q.repeat_interleave(spp, dim=0)  # noqa: E731
    d = rep(t1) * u[:, None] + rep(t2) * v[:, None] + rep(z) * w[:, None]
    return rep(p), d / d.norm(dim=1, keepdim=True)


def _woop64(v, i):
    """World-to-triangle transforms: (m, 3, 4) rows giving u, v and height."""
    a, b, c = (v.double()[i[:, k].long()] for k in range(3))
    e0, e1 = a - c, b - c
    M = torch.stack([e0, e1, torch.linalg.cross(e0, e1)], dim=2)
    M = M[torch.linalg.det(M) != 0]
    c = c[torch.linalg.det(torch.stack([e0, e1, torch.linalg.cross(e0, e1)], dim=2)) != 0]
    R = torch.linalg.inv(M)
    return torch.cat([R, -(R @ c[:, :, None])], dim=2)


def _all_hits(o, d, rows, tmin, tmax):
    """Closest t, u, v of each ray by testing every triangle (t = tmax and
    u = v = 0 on a miss)."""
    n, m = o.shape[0], rows.shape[0]
    out = [torch.empty(n, dtype=torch.float64, device=o.device) for _ in range(3)]
    flat = rows.reshape(3 * m, 4).T.contiguous()
    step = max(1, 60000000 // m)
    for at in range(0, n, step):
        O = (o[at:at + step] @ flat[:3] + flat[3]).reshape(-1, m, 3)
        D = (d[at:at + step] @ flat[:3]).reshape(-1, m, 3)
        t = -O[:, :, 2] / D[:, :, 2]
        u, v = O[:, :, 0] + t * D[:, :, 0], O[:, :, 1] + t * D[:, :, 1]
        ok = (t > tmin) & (t < tmax) & (u >= 0) & (v >= 0) & (u + v <= 1)
        best, k = torch.where(ok, t, torch.inf).min(dim=1)
        hit = torch.isfinite(best)
        out[0][at:at + step] = torch.where(hit, best, tmax)
        for q, x in ((1, u), (2, v)):
            out[q][at:at + step] = torch.where(hit, x.gather(1, k[:, None])[:, 0], 0.0)
    return out


def _f32(x):
    return float(np.float32(x))


def _ao64(v, i, pos, nrm, spp, seed, diag):
    o, d = _aorays64(pos, nrm, spp, seed)
    tmax = _f32(0.1 * diag)
    t = _all_hits(o, d, _woop64(v, i), _f32(1e-4 * diag), tmax)[0]
    return (t < tmax).double().reshape(-1, spp).mean(dim=1)


def exact(case, seed):
    path = case["path"]
    pairs = _rays(case) * (case["tris"] if "tris" in case else 1e9)
    if path not in ("bake", "closest", "build", "serve") or case.get("fused") or pairs > _TESTS:
        return None
    s = prepare(case, seed)
    if path == "closest":
        ds, r = s["ds"], s["rays"].double()
        t, u, v = _all_hits(r[:, :3], r[:, 4:7], _woop64(ds.vertices, ds.indices), float(r[0, 3]), float(r[0, 7]))
        return {"t": t, "u": u, "v": v}
    if path == "serve":
        got = []
        for k, (_, host, d, rs, _) in enumerate(s["requests"]):
            V, I = W.scene_of_size(1000 * seed + k % case["scenes"], case["tris"])
            pos, nrm = (torch.from_numpy(x).cuda() for x in host[:2])
            got.append(_ao64(torch.from_numpy(V).cuda(), torch.from_numpy(I).cuda(), pos, nrm, case["spp"], rs, d))
        return got
    v, i, d = (s["v"], s["i"], s["diag"]) if path == "build" else (s["ds"].vertices, s["ds"].indices, s["ds"].diag)
    return {"ao": _ao64(v, i, s["pos"], s["nrm"], case["spp"], seed, d)}
