"""What a program does with this library, as cases that can be timed.

Each case is one kind of call at one size: bulk traces of ray buffers, batched
jobs over many scenes, the host-buffer paths (pipeline, server), frames of the
integrators and the film.  A program keeps its scene, BVH, tracer and
integrator over many calls, so those are made once per scene and shared; rays,
cameras, sample keys and film samples are made from the seed and differ from
state to state.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import renderbox2_b200 as rb
from renderbox2_b200 import configs
from renderbox2_b200.accel import Platform
from renderbox2_b200.render import (AmbientOcclusionIntegratorParams, BidirectionalPathIntegratorLvcParams,
                                    DeviceScene, Filter, Integrator, IntersectionBuffer, PathIntegratorParams,
                                    film_develop, trace_isect)
from renderbox2_b200.serve import JobList, Server, build_pool

ORDERS = {"dfs": rb.NODE_ORDER_DFS, "bfs": rb.NODE_ORDER_BFS, "cw8": rb.NODE_ORDER_CW8}


def listed():
    return [
        # A query of a few thousand rays against a small scene: picking, collision or visibility
        # tests between other work, where the call itself is the cost.
        dict(name="trace_small", kind="trace", scene="heightfield", tris=2816, order="dfs", mode="closest", rays=8192),
        # A ray buffer of a million incoherent rays through the tracer as it is created.
        dict(name="trace_closest", kind="trace", scene="heightfield", tris=131840, order="dfs", mode="closest",
             rays=1 << 20),
        # Visibility of a million point pairs in a large scene, in the layout made for incoherent rays.
        dict(name="trace_occlusion", kind="trace", scene="heightfield", tris=500000, order="cw8", mode="occlusion",
             rays=1 << 20),
        # Full intersection records for a shading stage of the caller's own; not a round number of rays.
        dict(name="isect_records", kind="isect", scene="heightfield", tris=131840, order="dfs", mode="closest",
             rays=300007),
        # Many scenes, each with its own rays, as one graph-replayed launch (the batching workload's
        # launch configuration and spread of scene sizes, at a quarter of its scenes and rays).
        dict(name="batch_scenes", kind="batch", scenes=16, tri_min=1000, tri_max=500000, order="cw8", reorder=0,
             rays=1 << 18),
        # The same kind of jobs from pinned host buffers and back to them.
        dict(name="host_pipeline", kind="host", scenes=8, tri_min=1000, tri_max=131840, order="dfs", rays=1 << 19),
        # A burst of served requests: path-traced tiles and ray batches on resident scenes.
        dict(name="serve_burst", kind="serve", scenes=4, tri_min=1000, tri_max=100000, jobs=12, tile_max=320,
             rays_max=1 << 19),
        # An ambient occlusion frame (the configuration's own size).
        dict(name="ao_frame", kind="ao", scene="heightfield", tris=131840, order="cw8", width=512, height=512,
             samples=16, radius=0.1),
        # A preview tile of a path-traced image through the tracer as it is created.
        dict(name="pt_tile", kind="pt", scene="room", spheres=40, order="dfs", width=250, height=141, spp=4, depth=8,
             filter="none"),
        # A path-traced frame of a million triangles (the configuration's scene and film, a quarter of its samples).
        dict(name="pt_frame", kind="pt", scene="room", spheres=2000, order="cw8", width=1920, height=1080, spp=16,
             depth=8, filter="none"),
        # Bidirectional path tracing with the light-vertex cache (the configuration's film, a quarter of its samples).
        dict(name="bdpt_frame", kind="bdpt", scene="room", spheres=2000, order="cw8", width=1280, height=720, spp=4,
             length=6, connections=1),
        # Reconstruction of a film from its samples with the wide filter that renderers use by default.
        dict(name="film_gaussian", kind="film", filter="gaussian", xw=2.0, yw=2.0, width=1280, height=720, spp=16),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["trace", "trace", "isect", "batch", "batch", "host", "serve", "ao", "pt", "pt", "bdpt",
                       "film"])
    c = dict(kind=kind)
    if kind in ("trace", "isect", "ao"):
        c.update(scene="heightfield", tris=log_int(1000, 200000), order=rng.choice(["dfs", "bfs", "cw8"]))
    if kind in ("pt", "bdpt"):
        c.update(scene="room", spheres=log_int(10, 500), order=rng.choice(["dfs", "bfs", "cw8"]),
                 width=log_int(64, 1280), height=log_int(64, 720))
    if kind == "trace":
        c.update(mode=rng.choice(["closest", "occlusion"]), rays=log_int(1000, 1 << 20))
    elif kind == "isect":
        c.update(mode=rng.choice(["closest", "any"]), rays=log_int(1000, 1 << 20))
    elif kind == "batch":
        c.update(scenes=rng.randint(2, 12), tri_min=1000, tri_max=log_int(2000, 50000), rays=log_int(2000, 200000),
                 order=rng.choice(["bfs", "cw8", "cw8"]), reorder=rng.choice([0, 0, 4, 5]))
    elif kind == "host":
        c.update(scenes=rng.randint(1, 6), tri_min=1000, tri_max=log_int(2000, 50000), rays=log_int(5000, 400000),
                 order=rng.choice(["dfs", "cw8"]))
    elif kind == "serve":
        c.update(scenes=rng.randint(1, 4), tri_min=1000, tri_max=log_int(2000, 50000), jobs=rng.randint(2, 12),
                 tile_max=log_int(65, 320), rays_max=log_int(70000, 1 << 19))
    elif kind == "ao":
        c.update(width=log_int(64, 700), height=log_int(64, 512), samples=log_int(1, 16),
                 radius=round(rng.uniform(0.05, 0.5), 3))
    elif kind == "pt":
        c.update(spp=log_int(1, 16), depth=rng.randint(1, 8), filter=rng.choice(["none", "none", "gaussian"]))
    elif kind == "bdpt":
        c.update(spp=log_int(1, 4), length=rng.randint(3, 8), connections=rng.randint(1, 3))
    elif kind == "film":
        c.update(filter=rng.choice(["none", "box", "triangle", "gaussian"]), xw=round(rng.uniform(0.5, 3.0), 2),
                 yw=round(rng.uniform(0.5, 3.0), 2), width=log_int(64, 1280), height=log_int(64, 720),
                 spp=log_int(1, 16))
    return c


# ------------------------------------------------------- what a program keeps
@functools.lru_cache(maxsize=None)
def heightfield(seed, tris):
    scene = rb.heightfield_for_triangles(seed, tris)
    return scene, rb.BVH(scene, platform=Platform(configs.BUILD["sah_node_cost"], configs.BUILD["sah_triangle_cost"]))


@functools.lru_cache(maxsize=None)
def room(spheres):
    # The path tracing configuration's room; fewer spheres make it smaller.
    k = configs.CONFIG2
    scene = rb.RoomScene(seed=k["seed"], n_boxes=max(2, spheres // 20), n_spheres=spheres,
                         sphere_subdiv=k["sphere_subdiv"], rmin=k["rmin"], rmax=k["rmax"], n_lights=k["n_lights"],
                         emission=k["emission"], room_size=k["room_size"])
    return scene, rb.BVH(scene, platform=Platform(configs.BUILD["sah_node_cost"], configs.BUILD["sah_triangle_cost"]))


def scene_and_bvh(c):
    return room(c["spheres"]) if c["scene"] == "room" else heightfield(1, c["tris"])


@functools.lru_cache(maxsize=None)
def tracer_of(bvh, order):
    t = rb.CudaTracer(bvh)
    t.set_node_order(ORDERS[order])
    return t


@functools.lru_cache(maxsize=None)
def device_scene(scene):
    return DeviceScene(scene)


@functools.lru_cache(maxsize=None)
def integrator(scene, bvh, order):
    return Integrator(tracer_of(bvh, order), device_scene(scene))


@functools.lru_cache(maxsize=None)
def pipeline():
    return rb.HostPipeline()


@functools.lru_cache(maxsize=None)
def server(scenes, tri_min, tri_max, tile_max, rays_max):
    pool = build_pool(spread(scenes, tri_min, tri_max))
    return pool, Server(pool, slots=8, max_tile=tile_max, max_rays=rays_max)


def spread(n, lo, hi):
    """n scene sizes, evenly spread over their logarithm."""
    return [int(round(lo * (hi / lo) ** (k / max(1, n - 1)))) for k in range(n)]


def camera(c, seed):
    """The configuration's view of its scene, moved a little for each seed."""
    k = configs.CONFIG1 if c["scene"] == "heightfield" else configs.CONFIG2
    s = k.get("room_size", 1.0)
    rng = np.random.default_rng(seed)
    eye = [(x + d) * s for x, d in zip(k["eye"], rng.uniform(-0.015, 0.015, 3))]
    look = [(x + d) * s for x, d in zip(k["lookat"], rng.uniform(-0.1, 0.1, 3))]
    return rb.PerspectiveCamera(eye, look, k["up"], (c["width"], c["height"]), k["fov"])


def surface_rays(scene, seed, n):
    return rb.surface_rays(scene, seed, n)[0]


# ------------------------------------------------------------------ the cases
def prepare(case, seed):
    c, k = case, case["kind"]
    if k in ("trace", "isect"):
        scene, bvh = scene_and_bvh(c)
        st = dict(kind=k, mode=c["mode"], tracer=tracer_of(bvh, c["order"]),
                  rays=torch.from_numpy(surface_rays(scene, seed, c["rays"])).cuda())
        if k == "isect":
            fields = None if c["mode"] == "closest" else ("intersected",)
            st.update(scene=device_scene(scene), out=IntersectionBuffer(c["rays"], fields=fields))
        return st
    if k == "batch":
        n, jobs, split = c["rays"], [], c["rays"] // 2
        hits = torch.empty((c["scenes"] * split, 4), dtype=torch.int32, device="cuda")
        occ = torch.empty((c["scenes"] * (n - split),), dtype=torch.uint8, device="cuda")
        for i, t in enumerate(spread(c["scenes"], c["tri_min"], c["tri_max"])):
            scene, bvh = heightfield(10 + i, t)
            rays = torch.from_numpy(surface_rays(scene, seed * 1000 + i, n)).cuda()
            tr = tracer_of(bvh, c["order"])
            jobs.append((tr, rays[:split], rb.MODE_CLOSEST, hits[i * split:(i + 1) * split], None))
            jobs.append((tr, rays[split:], rb.MODE_OCCLUSION, occ[i * (n - split):(i + 1) * (n - split)], None))
        b = rb.TraceBatch(jobs)
        # What the autotuner keeps for the batching workload in each layout.
        cw8 = c["order"] == "cw8"
        b.set_config(node_order=ORDERS[c["order"]], block_threads=256, regs=64 if cw8 else 48,
                     fetch_threshold=24 if cw8 else 8, chunk=4, node_threshold=12 if cw8 else 8,
                     reorder=c["reorder"])
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            b.capture(s)
        return dict(kind=k, batch=b, hits=hits, occ=occ)
    if k == "host":
        n, jobs, split = c["rays"], [], c["rays"] // 2
        hits = torch.empty((c["scenes"] * split, 4), dtype=torch.int32).pin_memory()
        occ = torch.empty((c["scenes"] * (n - split),), dtype=torch.uint8).pin_memory()
        for i, t in enumerate(spread(c["scenes"], c["tri_min"], c["tri_max"])):
            scene, bvh = heightfield(10 + i, t)
            rays = torch.from_numpy(surface_rays(scene, seed * 1000 + i, n)).pin_memory()
            tr = tracer_of(bvh, c["order"])
            jobs.append((tr, rays[:split], rb.MODE_CLOSEST, hits[i * split:(i + 1) * split], None))
            jobs.append((tr, rays[split:], rb.MODE_OCCLUSION, occ[i * (n - split):(i + 1) * (n - split)], None))
        return dict(kind=k, pipe=pipeline(), keep=jobs, jobs=rb.HostPipeline.job_array(jobs), hits=hits, occ=occ)
    if k == "serve":
        pool, srv = server(c["scenes"], c["tri_min"], c["tri_max"], c["tile_max"], c["rays_max"])
        jl, rng = JobList(), np.random.default_rng(seed)
        for j in range(c["jobs"]):
            # Two tiles for each ray batch, as in the serving mix; sizes evenly spread so that
            # every seed has the same work.
            b, f = j % c["scenes"], (j // 3 + 0.5) / max(1, c["jobs"] / 3)
            if j % 3 < 2:
                ex, ez = rng.uniform(0.2, 0.8, 2)
                jl.add_tile(b, int(64 + (c["tile_max"] - 64) * min(1.0, f)), (1, 4, 16)[(j // 3) % 3],
                            seed=int(rng.integers(1 << 31)), eye=(-ex, 0.9, ez - 0.9), lookat=(-ex, 0.0, ez))
            else:
                n = int(65536 * (c["rays_max"] / 65536) ** min(1.0, f))
                jl.add_rays(b, surface_rays(pool.scenes[b], int(rng.integers(1 << 31)), n),
                            rb.MODE_CLOSEST if (j // 3) % 2 == 0 else rb.MODE_OCCLUSION)
        return dict(kind=k, server=srv, jobs=jl)
    if k == "film":
        g = torch.Generator(device="cuda").manual_seed(seed)
        w, h, spp = c["width"], c["height"], c["spp"]
        p = torch.arange(w * h, device="cuda")
        base = torch.stack([p % w, p // w], 1).float().repeat(spp, 1)
        xy = base + torch.rand((spp * w * h, 2), generator=g, device="cuda") * 0.999
        L = torch.empty((spp * w * h, 4), device="cuda").exponential_(1.0, generator=g)
        return dict(kind=k, filter=film_filter(c), size=(w, h, spp), xy=xy, L=L)
    scene, bvh = scene_and_bvh(c)
    st = dict(kind=k, it=integrator(scene, bvh, c["order"]), camera=camera(c, seed))
    if k == "ao":
        st["params"] = AmbientOcclusionIntegratorParams(samples=c["samples"], radius=c["radius"], seed=seed)
    elif k == "pt":
        st["params"] = PathIntegratorParams(spp=c["spp"], max_depth=c["depth"], rr_start=3, rr_prob=0.95, seed=seed)
        st["filter"] = None if c["filter"] == "none" else Filter("gaussian", 2.0, 2.0, 2.0)
    else:
        st["params"] = BidirectionalPathIntegratorLvcParams(spp=c["spp"], max_path_length=c["length"],
                                                            connections=c["connections"], seed=seed)
    return st


def film_filter(c):
    return Filter(c["filter"], c["xw"], c["yw"], 2.0)


def run(st):
    k = st["kind"]
    if k == "trace":
        if st["mode"] == "occlusion":
            return st["tracer"].trace_occlusion(st["rays"])
        return rb.hits_view(st["tracer"].trace(st["rays"]))
    if k == "isect":
        return dict(trace_isect(st["tracer"], st["scene"], st["rays"], any_hit=st["mode"] == "any", out=st["out"]).t)
    if k == "batch":
        st["batch"].launch()
        return [rb.hits_view(st["hits"]), st["occ"]]
    if k == "host":
        st["pipe"].trace_jobs(st["jobs"])
        return [rb.hits_view(st["hits"]), st["occ"]]
    if k == "serve":
        st["server"].run(st["jobs"])
        return [rb.hits_view(o) if o.dtype == torch.int32 else o for o in st["jobs"].outputs]
    if k == "film":
        return film_develop(st["filter"], *st["size"], st["xy"], st["L"])
    it, cam, p = st["it"], st["camera"], st["params"]
    if k == "ao":
        return it.render_ao(cam, p)
    if k == "pt":
        it.set_filter(st["filter"])
        return it.render_pt(cam, p)
    return it.render_bdpt(cam, p)


def work(case):
    """Rays in, records out, and the scene's triangles once (at most one per ray); per ray one root-to-leaf walk
    of box pairs and one triangle test.  Frames read no rays: their image is the output, their rays are counted
    as operations only."""
    c, k = case, case["kind"]
    if k == "film":
        n, taps = c["width"] * c["height"] * c["spp"], (1 if c["filter"] == "none" else 4 * c["xw"] * c["yw"])
        return {"bytes": n * (16 + (0 if c["filter"] == "none" else 8)) + 12 * c["width"] * c["height"],
                "flops": n * 8 * max(1.0, taps)}
    if k in ("batch", "host"):
        sizes, n = spread(c["scenes"], c["tri_min"], c["tri_max"]), c["rays"]
        return {"bytes": sum(n * 32 + n // 2 * 17 + 48 * min(n, t) for t in sizes),
                "flops": sum(n * walk(t) for t in sizes)}
    if k == "serve":
        t, groups = c["tri_max"], max(1, c["jobs"] // 3)
        rays, tiles = groups * (65536 * c["rays_max"]) ** 0.5, 2 * groups * (0.5 * (64 + c["tile_max"])) ** 2
        return {"bytes": rays * 41 + tiles * 12, "flops": (rays + tiles * 7 * 4) * walk(t)}
    t = c["tris"] if c["scene"] == "heightfield" else 500 * c["spheres"]
    if k in ("trace", "isect"):
        out = {"occlusion": 1, "any": 1, "closest": 16 if k == "trace" else 71}[c["mode"]]
        return {"bytes": c["rays"] * (32 + out) + 48 * min(t, c["rays"]), "flops": c["rays"] * walk(t)}
    npix = c["width"] * c["height"]
    if k == "ao":
        return {"bytes": npix * 4 + 48 * t, "flops": npix * (1 + c["samples"]) * walk(t)}
    rays = 2 * min(c["depth"], 4) if k == "pt" else 3 * min(c["length"], 4)
    return {"bytes": npix * 12 + 48 * t, "flops": npix * c["spp"] * rays * walk(t)}


def walk(tris):
    return 48 * math.log2(max(2, tris)) + 60


# -------------------------------------------------------------- in 64 bits
def exact(case, seed):
    c, k = case, case["kind"]
    if k == "film":
        return exact_film(c, seed)
    if k in ("trace", "isect") and c["mode"] == "closest" and c["rays"] * c["tris"] <= 1.5e11:
        return exact_hits(c, seed)
    return None  # an exhaustive search over every ray and triangle of the others takes minutes to hours


def exact_film(c, seed):
    s = prepare(c, seed)
    w, h, spp = s["size"]
    L = s["L"].double().view(spp, h, w, 4)[..., :3]
    if c["filter"] == "none":
        return L.mean(0).reshape(-1, 3)
    xy = s["xy"].double().view(spp, h, w, 2) - 0.5
    xw, yw = c["xw"], c["yw"]
    y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")

    def table(n):  # the film's 16 entries per axis
        t = (torch.arange(16, device="cuda").double() + 0.5) * n / 16
        if c["filter"] == "triangle":
            return n - t
        if c["filter"] == "gaussian":
            return (-2.0 * t * t).exp() - math.exp(-2.0 * n * n)
        return torch.ones_like(t)

    tx, ty = table(xw), table(yw)
    num = torch.zeros((h, w, 3), dtype=torch.float64, device="cuda")
    den = torch.zeros((h, w), dtype=torch.float64, device="cuda")
    rx, ry = int(xw + 0.5) + 1, int(yw + 0.5) + 1
    for oy in range(-ry, ry + 1):
        for ox in range(-rx, rx + 1):
            px, py = x + ox, y + oy  # the output pixel that the samples of (x, y) may reach
            ok = (px >= 0) & (px < w) & (py >= 0) & (py < h)
            dx, dy = px - xy[..., 0], py - xy[..., 1]
            inside = ok & (dx.abs() <= xw) & (dy.abs() <= yw)
            ix = (dx.abs() / xw * 16).long().clamp(max=15)
            iy = (dy.abs() / yw * 16).long().clamp(max=15)
            wt = torch.where(inside, tx[ix] * ty[iy], 0.0)
            at = (py.clamp(0, h - 1) * w + px.clamp(0, w - 1)).reshape(-1)
            num.view(-1, 3).index_add_(0, at, (wt[..., None] * L).sum(0).reshape(-1, 3))
            den.view(-1).index_add_(0, at, wt.sum(0).reshape(-1))
    return (num / torch.where(den > 0, den, 1.0)[..., None]).clamp(min=0).reshape(-1, 3)


def exact_hits(c, seed):
    """Every ray against every triangle (Moller and Trumbore, "Fast, Minimum Storage Ray/Triangle Intersection",
    1997); u and v are the weights of a triangle's first and second vertex."""
    scene = scene_and_bvh(c)[0]
    rays = torch.from_numpy(surface_rays(scene, seed, c["rays"])).cuda().double()
    v = torch.from_numpy(scene.vertices).cuda().double()[torch.from_numpy(scene.indices.astype(np.int64)).cuda()]
    a, e1, e2 = v[:, 2], v[:, 0] - v[:, 2], v[:, 1] - v[:, 2]
    n = torch.linalg.cross(e1, e2)
    an = (a * n).sum(1)
    # Scalar triple products as products of matrices: det = -d.n, and with m = o x d,
    # (o - a) x d . e = m . e - (a x d) . e = m . e + d . (a x e).
    ae1, ae2 = torch.linalg.cross(a, e1), torch.linalg.cross(a, e2)
    prim = torch.full((len(rays),), -1, dtype=torch.int64, device="cuda")
    step = max(1, int(4e8 / len(v)))
    for at in range(0, len(rays), step):
        r = rays[at:at + step]
        o, tmin, d, tmax = r[:, :3], r[:, 3:4], r[:, 4:7], r[:, 7:8]
        m = torch.linalg.cross(o, d)
        det = d @ n.T
        t = (an[None] - o @ n.T) / det
        bu = (m @ e2.T + d @ ae2.T) / -det
        bv = (m @ e1.T + d @ ae1.T) / det
        t = torch.where((bu >= 0) & (bv >= 0) & (bu + bv <= 1) & (t > tmin) & (t < tmax), t, math.inf)
        best, i = t.min(1)
        prim[at:at + step] = torch.where(best < math.inf, i, -1)
        del det, t, bu, bv
    hit, i = prim >= 0, prim.clamp(min=0)
    o, d = rays[:, :3], rays[:, 4:7]
    det = (d * n[i]).sum(1)
    s = o - a[i]
    t = torch.where(hit, -(s * n[i]).sum(1) / det, rays[:, 7])
    sd = torch.linalg.cross(s, d)
    zero = torch.zeros_like(t)
    bu = torch.where(hit, -(sd * e2[i]).sum(1) / det, zero)
    bv = torch.where(hit, (sd * e1[i]).sum(1) / det, zero)
    if c["kind"] == "trace":
        return [None, t, bu, bv]
    # Records of rays that miss are not written: they keep what the buffer was made with.
    nan = torch.full_like(t, math.nan)
    ng = n[i] / n[i].norm(dim=1, keepdim=True)

    def plane(x):
        return torch.where(hit[:, None], x, nan[:, None]).T.contiguous()

    return dict(position=plane(o + t[:, None] * d), geometric_normal=plane(ng), shading_normal=plane(ng),
                incoming_direction=plane(-d), uv=torch.where(hit[:, None], torch.stack([bu, bv], 1), nan[:, None]),
                epsilon=torch.where(hit, 1e-3 * t, nan))
