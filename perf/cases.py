"""Performance cases of the framework: the calls a program makes, over the range of sizes it makes them at.

Every case goes through the package's public entry points (Scene.trace, Scene.trace_host, Pool.trace,
Scene.render with accum_clear and resolve, build_bvh_device, Server.submit / wait).  `listed` names
the fixed cases, `draw` gives further ones from the same ranges, `prepare` makes what a program holds
before the call (scene handle, rays, output buffers), `run` is one pass, `work` counts what a pass
cannot do without and `exact` gives a pass's results in binary64 where brute force can.

Kinds:
  trace   a batch of device rays on one scene: a pick ray, camera rays, incoherent queries, shadow rays
  host    the same with rays and hits in page-locked host memory
  pool    many scenes, each with its own batch, in one call
  render  one frame: clear, path trace all samples, resolve
  build   the LBVH of triangles that are already on the device
  serve   a burst of requests against resident scenes of a server
"""
from __future__ import annotations

import math

import numpy as np
import torch

import raytracergpu_mastersproject_gb300 as rt

# Ranges of `listed` and `draw`: triangles of a scene, rays of a call.
TRIS = (256, 4_194_304)
RAYS = (1, 16_777_216)
SIGMA = 0.002  # vertex spread of the soups, in units of a cube with 4,194,304 triangles
INF = float("inf")


def listed():
    return [
        # a mouse pick or a line-of-sight probe: a handful of rays, latency is all there is
        dict(name="pick", kind="trace", scene="mesh", tris=20_482, rays=17, any=False, sort=False, camera=False),
        # the primary rays of a 640x360 view of a 20,482-triangle mesh (the camera workload of the tests)
        dict(name="camera", kind="trace", scene="mesh", tris=20_482, rays=230_400, width=640, any=False, sort=False,
             camera=True),
        # shadow and visibility rays, any hit, in the order the program made them
        dict(name="shadow", kind="trace", scene="soup", tris=262_144, rays=1_000_003, any=True, sort=False,
             camera=False),
        # an ordinary incoherent batch (one bounce of a small frame), reordered by the library
        dict(name="bounce", kind="trace", scene="soup", tris=1_048_576, rays=100_003, any=False, sort=True,
             camera=False),
        # the largest batch: 16.8 M incoherent rays on 4.2 M triangles (the headline workload)
        dict(name="soup_large", kind="trace", scene="soup", tris=4_194_304, rays=16_777_216, any=False, sort=True,
             camera=False),
        # rays and hits in page-locked host memory: copies and tracing in one call
        dict(name="host", kind="host", scene="soup", tris=524_288, rays=3_000_002, any=False, sort=True),
        # many scenes of uneven size, each with its own batch (the batched workload at 64 scenes)
        dict(name="pool", kind="pool", scenes=64, tris_lo=1_000, tris_hi=64_000, rays_lo=4_000, rays_hi=256_000,
             any=False),
        # a full frame: 64 displaced spheres (5.2 M triangles), 1280x720, 16 samples, depth 8
        dict(name="frame", kind="render", spheres=64, subdiv=6, width=1280, height=720, spp=16, depth=8,
             extended=True),
        # an interactive preview: small odd-sized image, one sample, the reference's shading
        dict(name="preview", kind="render", spheres=12, subdiv=4, width=317, height=179, spp=1, depth=4,
             extended=False),
        # the LBVH of a small dynamic scene, rebuilt every frame
        dict(name="build_small", kind="build", scene="mesh", tris=20_482),
        # the LBVH of a large scene
        dict(name="build_large", kind="build", scene="soup", tris=4_194_304),
        # a burst of queries of 1 K to 128 K rays against eight resident scenes
        dict(name="serve", kind="serve", scenes=8, tris_lo=16_000, tris_hi=256_000, requests=24, rays_lo=1_000,
             rays_hi=128_000),
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | 1 if n > 2 and n < hi and rng.random() < 0.6 else n))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "host", "pool", "render", "build", "build", "serve"])
    if kind == "trace":
        if rng.random() < 0.25:  # camera rays of a mesh
            w, h = rng.randint(33, 1280), rng.randint(17, 720)
            return dict(kind=kind, scene="mesh", tris=20 * 4 ** rng.randint(2, 6) + 2, rays=w * h, width=w,
                        any=rng.random() < 0.3, sort=False, camera=True)
        return dict(kind=kind, scene=rng.choice(["mesh", "soup", "soup"]) if rng.random() < 0.5 else "soup",
                    tris=_log_int(rng, *TRIS), rays=_log_int(rng, RAYS[0], RAYS[1] // 2), any=rng.random() < 0.35,
                    sort=rng.random() < 0.5, camera=False)
    if kind == "host":
        # An odd count of more than 524,288 rays is left out: it takes two staging chunks, and versions that put
        # the second one straight after the first read it off its alignment.
        rays = _log_int(rng, 256, 8_388_608)
        return dict(kind=kind, scene="soup", tris=_log_int(rng, 1_000, 1_048_576),
                    rays=rays & ~1 if rays > 524_288 else rays, any=rng.random() < 0.3, sort=rng.random() < 0.6)
    if kind == "pool":
        lo, rays = _log_int(rng, 256, 8_000), _log_int(rng, 256, 16_000)
        return dict(kind=kind, scenes=rng.randint(2, 96), tris_lo=lo, tris_hi=lo * rng.randint(2, 16), rays_lo=rays,
                    rays_hi=rays * rng.randint(2, 16), any=rng.random() < 0.3)
    if kind == "render":
        return dict(kind=kind, spheres=rng.randint(4, 64), subdiv=rng.randint(2, 5), width=rng.randint(64, 1280),
                    height=rng.randint(48, 720), spp=_log_int(rng, 1, 16), depth=rng.randint(2, 12),
                    extended=rng.random() < 0.6)
    if kind == "build":
        return dict(kind=kind, scene="soup", tris=_log_int(rng, 2, TRIS[1]))
    lo, rays = _log_int(rng, 1_000, 32_000), _log_int(rng, 500, 16_000)
    return dict(kind=kind, scenes=rng.randint(2, 12), tris_lo=lo, tris_hi=lo * rng.randint(2, 12),
                requests=rng.randint(2, 48), rays_lo=rays, rays_hi=rays * rng.randint(2, 16))


# ------------------------------------------------------------------ inputs
def _soup(seed, stream, n):
    """n triangles at the headline workload's density, in a cube of side (n / 4,194,304)^(1/3)."""
    side = (n / 4_194_304) ** (1.0 / 3.0)
    return rt.gen_soup(seed, stream, n, side, SIGMA), side


def _mesh(n):
    """A sphere of about n triangles on a ground quad; n = 20 * 4^k + 2 gives the whole sphere."""
    k = 0
    while 20 * 4 ** k + 2 < n:
        k += 1
    ground = rt.gen_config1()[0][-2:]
    tris = np.concatenate([rt.gen_icosphere(k, (0.0, 0.0, 0.0), 1.0, 0), ground])
    return tris[len(tris) - max(n, 2):]


def _camera(seed, width, height, num_triangles):
    r = np.random.RandomState(seed % (1 << 32))
    a, y = r.uniform(0.0, 2.0 * math.pi), r.uniform(0.3, 1.2)
    ubo = rt.make_ubo((4.0 * math.sin(a), y, 4.0 * math.cos(a)), (0.0, 0.0, 0.0), fov=60.0, depth=8,
                      num_triangles=num_triangles)
    return rt.gen_camera_rays(ubo, width, height)


def _geometry(case, seed):
    """-> (triangles, rays) of a trace or host case."""
    if case["scene"] == "mesh":
        tris = _mesh(case["tris"])
        if case["camera"]:
            return tris, _camera(seed, case["width"], case["rays"] // case["width"], len(tris))
        rays = rt.gen_rays(seed, 0, case["rays"], 4.0, 1e-4, INF)  # origins around the sphere
        rays["org"] -= np.float32([2.0, 0.5, 2.0])
        return tris, rays
    tris, side = _soup(seed, 0, case["tris"])
    return tris, rt.gen_rays(seed, 0, case["rays"], side, 1e-4, INF)


def _log_sizes(lo, hi, count):
    """Sizes spread evenly over the logarithm of [lo, hi]; most come out odd or ragged."""
    return [int(v) for v in np.rint(np.exp(np.linspace(math.log(lo), math.log(hi), count)))]


def _batches(case, seed):
    """-> (soups, [(scene, rays)]) of a pool or serve case; the seed decides which scene and batch go together."""
    r = np.random.RandomState(seed % (1 << 32))
    nt = _log_sizes(case["tris_lo"], case["tris_hi"], case["scenes"])
    count = case["scenes"] if case["kind"] == "pool" else case["requests"]
    nr = [int(v) for v in r.permutation(_log_sizes(case["rays_lo"], case["rays_hi"], count))]
    where = list(range(count)) if case["kind"] == "pool" else [int(v) for v in r.randint(0, case["scenes"], count)]
    soups = [_soup(seed, i + 1, n) for i, n in enumerate(nt)]
    return [t for t, _ in soups], [(w, rt.gen_rays(seed, 1000 + i, n, soups[w][1], 1e-4, INF))
                                   for i, (w, n) in enumerate(zip(where, nr))]


def _cuda(a):
    return torch.from_numpy(a.view(np.uint8).reshape(-1)).cuda()


def _hits(h, any_hit):
    """What a program takes from a hit buffer of int32 [n, 2]; any hit promises no particular primitive."""
    return {"hit": h[:, 0]} if any_hit else {"prim": h[:, 0], "t": h.view(torch.float32)[:, 1]}


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("trace", "host"):
        tris, rays = _geometry(case, seed)
        st["scene"] = rt.Scene(tris)
        if kind == "trace":
            st["rays"] = _cuda(rays)
            st["hits"] = torch.empty((len(rays), 2), dtype=torch.int32, device="cuda")
        else:
            pin = torch.empty(rays.nbytes, dtype=torch.uint8, pin_memory=True)
            pin.numpy()[:] = rays.view(np.uint8).reshape(-1)
            st["keep"] = pin
            st["rays"] = pin.numpy().view(rt.RAY_DTYPE)
            st["hits"] = torch.empty((len(rays), 2), dtype=torch.int32, pin_memory=True)
            st["hits_np"] = st["hits"].numpy().reshape(-1).view(rt.HIT_DTYPE)
        st["out"] = _hits(st["hits"], case["any"])
    elif kind in ("pool", "serve"):
        soups, batches = _batches(case, seed)
        count = len(batches)
        at = [int(v) for v in np.concatenate([[0], np.cumsum([len(b) for _, b in batches])])]
        rays = np.concatenate([b for _, b in batches])
        if kind == "pool":
            st["pool"] = rt.Pool()
            ids = [st["pool"].add_scene(t) for t in soups]
            st["rays"] = _cuda(rays).view(-1, 32)
            st["hits"] = torch.empty((len(rays), 2), dtype=torch.int32, device="cuda")
            st["jobs"] = [(ids[batches[i][0]], st["rays"][at[i]:at[i + 1]], st["hits"][at[i]:at[i + 1]])
                          for i in range(count)]
            st["out"] = _hits(st["hits"], case["any"])
        else:
            st["server"] = rt.Server(stage_rays=1 << 23)
            ups = [st["server"].upload(t) for t in soups]
            ids = [st["server"].wait(u).scene_id for u in ups]
            pin = torch.empty(rays.nbytes, dtype=torch.uint8, pin_memory=True)
            pin.numpy()[:] = rays.view(np.uint8).reshape(-1)
            st["keep"] = pin
            h_rays = pin.numpy().view(rt.RAY_DTYPE)
            st["hits"] = torch.empty((len(rays), 2), dtype=torch.int32, pin_memory=True)
            h_hits = st["hits"].numpy().reshape(-1).view(rt.HIT_DTYPE)
            st["requests"] = [(ids[batches[i][0]], h_rays[at[i]:at[i + 1]], h_hits[at[i]:at[i + 1]])
                              for i in range(count)]
            st["out"] = _hits(st["hits"], False)
    elif kind == "render":
        tris, mats = rt.gen_spheres_scene(seed, case["spheres"], case["subdiv"], 0.05)
        if not case["extended"]:  # the reference's shading scatters diffuse surfaces and ends on lights
            mats["materialType"] = rt.MAT_DIFFUSE
            mats["materialType"][::4] = rt.MAT_LIGHT
        w, h = case["width"], case["height"]
        st["scene"] = rt.Scene(tris, materials=mats)
        st["ubo"] = rt.make_ubo((0.0, 3.0, 28.0), (0.0, 0.0, 0.0), fov=40.0, depth=case["depth"],
                                random_state=seed % 100_000, num_triangles=len(tris), num_materials=len(mats))
        st["accum"] = torch.empty(w * h * 4, dtype=torch.float32, device="cuda")
        st["image"] = torch.empty(w * h * 4, dtype=torch.float32, device="cuda")
        st["out"] = {"accum": st["accum"], "image": st["image"]}
    else:
        tris = _mesh(case["tris"]) if case["scene"] == "mesh" else _soup(seed, 0, case["tris"])[0]
        if case["scene"] == "mesh":  # a moving object: the same sphere, elsewhere
            shift = np.random.RandomState(seed % (1 << 32)).uniform(-3.0, 3.0, 3).astype(np.float32)
            for v in ("v0", "v1", "v2"):
                tris[v][:-2, :3] += shift
        st["count"] = len(tris)
        st["tris"] = _cuda(tris)
        st["nodes"] = torch.empty(((2 * len(tris) - 1) * 10,), dtype=torch.int32, device="cuda")
        st["out"] = {"nodes": st["nodes"]}
    return st


# --------------------------------------------------------------------- run
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "trace":
        st["scene"].trace(st["rays"], st["hits"], any_hit=case["any"], sort=case["sort"])
    elif kind == "host":
        st["scene"].trace_host(st["rays"], any_hit=case["any"], out=st["hits_np"], sort=case["sort"])
    elif kind == "pool":
        st["pool"].trace(st["jobs"], any_hit=case["any"])
    elif kind == "render":
        w, h = case["width"], case["height"]
        rt.accum_clear(st["accum"], w, h)
        st["scene"].render(st["ubo"], st["accum"], w, h, case["spp"],
                           shade_mode=rt.SHADE_EXTENDED if case["extended"] else rt.SHADE_REFERENCE,
                           background=(0.6, 0.7, 1.0))
        rt.resolve(st["accum"], w, h, case["spp"], st["image"])
    elif kind == "build":
        rt.build_bvh_device(st["tris"], st["count"], d_nodes=st["nodes"])
    else:
        server = st["server"]
        ids = [server.submit(sid, rays, hits) for sid, rays, hits in st["requests"]]
        for i in ids:
            server.wait(i)
    if "hit" in st["out"]:  # any hit answers yes or no
        return {"hit": st["out"]["hit"] != -1}
    return st["out"]


# -------------------------------------------------------------------- work
def _query_flops(tris):
    """Two box tests a level of a balanced binary tree (18 operations each) and one triangle test (60)."""
    return 36.0 * max(1.0, math.log2(max(tris, 2))) + 60.0


def work(case):
    kind = case["kind"]
    if kind in ("trace", "host"):
        n, t = case["rays"], case["tris"]
        return {"bytes": 40.0 * n + 48.0 * min(t, 4 * n), "flops": n * _query_flops(t)}
    if kind in ("pool", "serve"):
        n = sum(_log_sizes(case["rays_lo"], case["rays_hi"], case["scenes"] if kind == "pool" else case["requests"]))
        t = sum(_log_sizes(case["tris_lo"], case["tris_hi"], case["scenes"]))
        return {"bytes": 40.0 * n + 48.0 * t, "flops": n * _query_flops(t / case["scenes"])}
    if kind == "render":
        px = case["width"] * case["height"]
        t = case["spheres"] * 20 * 4 ** case["subdiv"]
        paths = px * case["spp"]
        return {"bytes": 32.0 * px + 48.0 * min(t, paths), "flops": (px + 0.4 * paths) * _query_flops(t) + 100.0 * paths}
    t = case["tris"]
    return {"bytes": 48.0 * t + 40.0 * (2 * t - 1), "flops": 60.0 * t}


# ------------------------------------------------------------------- exact
def _brute(tris, rays, dev):
    """Closest hits by brute force in binary64 (the plane and barycentric test of raytraceBVH.comp:118-149)."""
    f64 = lambda a: torch.from_numpy(np.ascontiguousarray(a).astype(np.float64)).to(dev)  # noqa: E731
    v0, v1, v2 = (f64(tris[k][:, :3]) for k in ("v0", "v1", "v2"))
    org, d = f64(rays["org"]), f64(rays["dir"])
    tmin, tmax = f64(rays["tmin"]), f64(rays["tmax"])
    u, v = v1 - v0, v2 - v0
    big = torch.linalg.cross(u, v)
    n = big / big.norm(dim=1, keepdim=True)
    w = big / (big * big).sum(dim=1, keepdim=True)
    plane = (n * v0).sum(dim=1)
    # a = w . (q x v) = q . (v x w) and b = w . (u x q) = q . (w x u), with q = p - v0
    ka, kb = torch.linalg.cross(v, w), torch.linalg.cross(w, u)
    a0, b0 = (ka * v0).sum(dim=1), (kb * v0).sum(dim=1)
    best = torch.full((len(rays),), INF, dtype=torch.float64, device=dev)
    prim = torch.full((len(rays),), -1, dtype=torch.int64, device=dev)
    step = max(1, 64_000_000 // max(1, len(tris)))
    for s in range(0, len(rays), step):
        o, e = org[s:s + step], d[s:s + step]
        den = e @ n.T
        t = (plane - o @ n.T) / den
        a = o @ ka.T + t * (e @ ka.T) - a0
        b = o @ kb.T + t * (e @ kb.T) - b0
        ok = (den.abs() >= 1e-4) & (t >= tmin[s:s + step, None]) & (t <= tmax[s:s + step, None])
        ok &= (a >= 0) & (b >= 0) & (a + b <= 1)
        t = torch.where(ok, t, torch.full_like(t, INF))
        m, k = t.min(dim=1)
        best[s:s + step] = m
        prim[s:s + step] = torch.where(torch.isinf(m), torch.full_like(k, -1), k)
    return prim, best


def exact(case, seed):
    """The hits of a closest-hit case in binary64, where testing every ray against every triangle is affordable.
    Any-hit answers and node arrays are whole numbers; a path-traced frame follows binary32 random numbers."""
    kind = case["kind"]
    if kind in ("render", "build") or case.get("any"):
        return None
    if kind in ("trace", "host"):
        if case["tris"] * case["rays"] > 6_000_000_000:
            return None
        tris, rays = _geometry(case, seed)
        pairs = [(tris, rays)]
    else:
        count = case["scenes"] if kind == "pool" else case["requests"]
        if case["tris_hi"] * sum(_log_sizes(case["rays_lo"], case["rays_hi"], count)) > 20_000_000_000:
            return None
        soups, batches = _batches(case, seed)
        pairs = [(soups[w], rays) for w, rays in batches]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    got = [_brute(tris, rays, dev) for tris, rays in pairs]
    return {"prim": torch.cat([g[0] for g in got]), "t": torch.cat([g[1] for g in got])}
