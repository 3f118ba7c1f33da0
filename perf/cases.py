"""Performance cases of the photon mapper: what a user's program has it do.

Every case is one pass through the public entry points (the Python classes of
photon_mapping_b200, and the C ABI's device-pointer calls for data that
already lies on the GPU). Kinds of case, and what each stands for:

  knn       PhotonMap.query_knn on host arrays: nearest-photon lists with
            their distances (a density or debugging view of the map, or a host
            integrator that asks for a few points at a time).
  radiance  the photon-map radiance estimate on an existing map, through
            PhotonMap.radiance (host arrays) or pm_photonmap_radiance_device
            (device tensors): primary hits of a frame in pixel order, or
            hit points in no order.
  rebuild   pm_photonmap_build_device followed by an estimate: a program that
            makes its own photons on the GPU and rebuilds its map per frame.
  frame     PhotonMapping.build + render: one frame with freshly traced photon
            maps, the loop of the renderer's own example program.
  batch     BatchRenderer.render + image: many small scenes in one step.
  gradient  DiffRenderer.forward + backward: one optimisation step over the
            scene's albedos and emission.
  scene     Scene.build + intersect: a new mesh and its camera's closest hits.

Sizes come from the render settings in photon_mapping_b200/configs.py, the
batched and gradient workloads of bench.py and the tests' small sets.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from photon_mapping_b200 import Context, PhotonMap
from photon_mapping_b200 import configs
from photon_mapping_b200 import scene as S
from photon_mapping_b200 import workloads as W
from photon_mapping_b200.batch import BatchRenderer, random_scene
from photon_mapping_b200.differentiable import DiffRenderer, perturbed_parameters
from photon_mapping_b200.integrator import PhotonMapping

MAX_DEPTH = configs.MAX_DEPTH
STORED_PER_EMITTED = 3.26  # photons a Cornell trace stores per photon emitted
# camera queries taken per ray of a frame of the room (0.873 of the rays end
# on a surface that is not the light): the same number whatever the jitter
HITS_PER_RAY = 0.85


def listed():
    return [
        # the smallest call: a host program asking for a few points
        dict(name="knn-64", kind="knn", photons="walls", n=20_000, nq=64, k=50),
        # a ragged host query set over a mid-sized map
        dict(name="knn-20k", kind="knn", photons="walls", n=300_007, nq=20_011, k=50),
        # small interactive estimate, host arrays in and out
        dict(name="radiance-2k-host", kind="radiance", photons="walls", n=200_000, queries="walls",
             nq=2_048, k=50, side=0, spp=0, host=True),
        # the benchmark's estimate: primary hits of a 512x512x4 frame on the
        # map of 1M emitted photons, everything on the GPU
        dict(name="radiance-room-1m", kind="radiance", photons="traced", n=1_000_000,
             queries="camera", nq=0, k=100, side=512, spp=4, host=False),
        # odd number of unordered hit points, large k
        dict(name="radiance-scattered-k300", kind="radiance", photons="cube", n=500_003,
             queries="walls", nq=65_537, k=300, side=0, spp=0, host=False),
        # the program's own photons, map rebuilt every frame
        dict(name="rebuild-1m", kind="rebuild", photons="walls", n=1_000_000, queries="walls",
             nq=65_536, k=50),
        # a small frame with the estimate at the first diffuse hit
        dict(name="frame-cornell-256", kind="frame", scene="cornell", photons=100_000, mult=1.0,
             width=256, height=256, spp=16, k=100, fg=0, n_gather=1),
        # final gathering with 16 gather rays per hit (the heaviest frame)
        dict(name="frame-cornell-512-gather16", kind="frame", scene="cornell", photons=1_000_000,
             mult=1.0, width=512, height=512, spp=4, k=100, fg=1, n_gather=16),
        # 563k triangles with mirror, glass and water; 1M global and 10M
        # caustics photons
        dict(name="frame-caustics-512", kind="frame", scene="caustics", photons=1_000_000,
             mult=10.0, width=512, height=512, spp=2, k=100, fg=1, n_gather=1),
        # many uneven scenes in one step
        dict(name="batch-8", kind="batch", scenes=8, first=0, tri_max=60_000, photons_max=1_000_000,
             side_max=512, spp=2),
        # one gradient step of the Cornell box
        dict(name="gradient-256", kind="gradient", photons=1_000_000, side=256, spp=16, k=50, fg=1),
        # a new mesh, and the closest hits of one camera frame
        dict(name="scene-250k", kind="scene", grid=354, side=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("knn", "radiance", "radiance", "radiance", "rebuild", "frame", "frame",
                       "batch", "gradient", "scene"))
    if kind == "knn":
        return dict(kind=kind, photons=rng.choice(("walls", "cube")), n=_log_int(rng, 1_000, 500_000),
                    nq=_log_int(rng, 1, 40_000), k=_log_int(rng, 4, 200))
    if kind == "radiance":
        if rng.random() < 0.5:
            return dict(kind=kind, photons="traced", n=_log_int(rng, 20_000, 1_000_000),
                        queries="camera", nq=0, k=_log_int(rng, 20, 200),
                        side=_log_int(rng, 48, 512), spp=rng.randint(1, 4),
                        host=rng.random() < 0.3)
        return dict(kind=kind, photons=rng.choice(("walls", "cube", "traced")),
                    n=_log_int(rng, 20_000, 1_000_000), queries="walls",
                    nq=_log_int(rng, 200, 300_000), k=_log_int(rng, 8, 400), side=0, spp=0,
                    host=rng.random() < 0.3)
    if kind == "rebuild":
        return dict(kind=kind, photons=rng.choice(("walls", "cube")), n=_log_int(rng, 5_000, 2_000_000),
                    queries="walls", nq=_log_int(rng, 1_000, 100_000), k=_log_int(rng, 8, 150))
    if kind == "frame":
        fg = rng.randint(0, 1)
        return dict(kind=kind, scene="cornell", photons=_log_int(rng, 20_000, 1_000_000), mult=1.0,
                    width=_log_int(rng, 64, 512), height=_log_int(rng, 64, 512),
                    spp=rng.randint(1, 4 if fg else 16), k=_log_int(rng, 20, 150), fg=fg,
                    n_gather=rng.randint(1, 12) if fg else 1)
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 7), first=rng.randint(8, 999), tri_max=_log_int(rng, 5_000, 60_000),
                    photons_max=_log_int(rng, 200_000, 1_000_000), side_max=_log_int(rng, 150, 512),
                    spp=rng.randint(1, 2))
    if kind == "gradient":
        return dict(kind=kind, photons=_log_int(rng, 50_000, 1_000_000), side=_log_int(rng, 48, 256),
                    spp=rng.randint(2, 16), k=_log_int(rng, 20, 100), fg=rng.randint(0, 1))
    return dict(kind=kind, grid=_log_int(rng, 30, 354), side=_log_int(rng, 32, 256))


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _mesh(kind):
    """The scene files of the frames; the same for every seed."""
    return configs.make_scene(kind)


@functools.lru_cache(maxsize=16)
def _batch_scene(i, tri_max, photons_max, side_max, spp):
    """Scene i of the batches and its settings; the seed draws its photons."""
    return random_scene(i, tri_range=(1_000, tri_max), photon_range=(50_000, photons_max),
                        side_range=(128, side_max), spp=spp, max_depth=MAX_DEPTH)


def _gen(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * stream + int(seed))


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float32)


def _wall_points(g, n):
    """n points on the Cornell walls: positions, inward normals, albedos."""
    w = torch.randint(0, len(W.WALLS), (n,), generator=g, device="cuda")
    pos = _rand(g, n, 3)
    axis = torch.tensor([x[0] for x in W.WALLS], device="cuda")[w]
    value = torch.tensor([x[1] for x in W.WALLS], device="cuda")[w]
    pos.scatter_(1, axis[:, None], value[:, None])
    normal = torch.tensor([x[2] for x in W.WALLS], device="cuda")[w]
    albedo = torch.tensor([x[3] for x in W.WALLS], device="cuda")[w]
    return pos, normal, albedo


def _hemisphere(g, normal):
    d = torch.nn.functional.normalize(
        torch.randn(normal.shape, generator=g, device="cuda", dtype=torch.float32), dim=1)
    return torch.where((d * normal).sum(1, keepdim=True) < 0, -d, d)


def _photons(kind, n, seed):
    """(n, 9) device photons: on the room's walls, or uniform in the cube."""
    g = _gen(seed, 1)
    if kind == "walls":
        pos, normal, albedo = _wall_points(g, n)
        wi = _hemisphere(g, normal)
        leak = _rand(g, n, 1) < 0.05  # arriving from below the surface
        return torch.cat([1.5 * _rand(g, n, 3) * albedo, pos, torch.where(leak, -wi, wi)], 1)
    wi = torch.nn.functional.normalize(
        torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float32), dim=1)
    return torch.cat([2.0 * _rand(g, n, 3), _rand(g, n, 3), wi], 1)


def _wall_queries(nq, seed):
    g = _gen(seed, 2)
    pos, normal, albedo = _wall_points(g, nq)
    wo = _hemisphere(g, normal)
    return torch.cat([pos, albedo[:, :1], wo, albedo[:, 1:2], normal, albedo[:, 2:]], 1).contiguous()


def _camera_rays(width, height, spp, seed):
    """Rays of a jittered frame in pixel order, sample-minor (host arrays)."""
    cam = configs.camera()
    vec = lambda a: torch.tensor(np.asarray(a, np.float32), device="cuda")  # noqa: E731
    n = width * height * spp
    jit = _rand(_gen(seed, 3), n, 2)
    pix = torch.arange(n, device="cuda") // spp
    u = (2.0 * (pix % width + jit[:, 0]) - width) / height
    v = (2.0 * (pix // width + jit[:, 1]) - height) / height
    sensor = vec(cam.position) + u[:, None] * vec(cam.right) + v[:, None] * vec(cam.up)
    pinhole = vec(cam.position) + float(cam.focal_length) * vec(cam.forward)
    d = torch.nn.functional.normalize(pinhole - sensor, dim=1)
    return sensor.cpu().numpy(), d.cpu().numpy()


def _scene_on(ctx, mesh):
    sc = S.Scene(ctx)
    sc.setMesh(mesh)
    sc.build()
    return sc


def _map_inputs(case, seed, ctx):
    """(photons (n, 9), queries (nq, 12)) as device tensors, and the number of
    photons emitted. A traced map is left built on ctx."""
    sc = None
    if case["photons"] == "traced" or case["queries"] == "camera":
        sc = _scene_on(ctx, _mesh("cornell"))
    if case["photons"] == "traced":
        pmi = PhotonMapping(case["n"], case["k"], 1.0, case["k"], 0, MAX_DEPTH, ctx=ctx)
        pmi.build(sc, seed=1 + seed)
        photons = None
    else:
        photons = _photons(case["photons"], case["n"], seed)
    if case["queries"] == "camera":
        o, d = _camera_rays(case["side"], case["side"], case["spp"], seed)
        q = W.hit_queries(sc.mesh, o, d, sc.intersect(o, d))[:_n_queries(case)]
        queries = torch.from_numpy(q).cuda()
    else:
        queries = _wall_queries(case["nq"], seed)
    return photons, queries


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "seed": int(seed)}
    if kind in ("knn", "radiance", "rebuild"):
        ctx = st["ctx"] = Context(0)
        pm = st["map"] = PhotonMap(ctx)
        if kind == "knn":
            pm.setPhotons(_photons(case["photons"], case["n"], seed).cpu().numpy())
            pm.build()
            st["queries"] = _wall_queries(case["nq"], seed)[:, :3].cpu().numpy()
            return st
        photons, queries = _map_inputs(case, seed, ctx)
        if kind == "radiance" and photons is not None:
            pm.setPhotons(photons.cpu().numpy())
            pm.build()
            photons = None
        st["photons"] = photons
        if case.get("host"):
            st["queries"] = queries.cpu().numpy()
        else:
            st["queries"] = queries
            st["out"] = torch.empty((queries.shape[0], 3), device="cuda")
    elif kind == "frame":
        ctx = st["ctx"] = Context(0)
        st["scene"] = _scene_on(ctx, _mesh(case["scene"]))
        st["camera"] = configs.camera()
        st["pmi"] = PhotonMapping(case["photons"], case["k"], case["mult"], case["k"], case["fg"],
                                  MAX_DEPTH, ctx=ctx)
    elif kind == "batch":
        scenes = []
        for i in range(case["scenes"]):
            sc = _batch_scene(case["first"] + i, case["tri_max"], case["photons_max"],
                              case["side_max"], case["spp"])
            scenes.append(dict(sc, seed=1000 * int(seed) + i))
        st["batch"] = BatchRenderer(scenes)
    elif kind == "gradient":
        ctx = st["ctx"] = Context(0)
        r = st["renderer"] = DiffRenderer(
            ctx, _mesh("cornell"), configs.camera(), case["side"], case["side"], case["spp"],
            case["photons"], case["k"], final_gathering_depth=case["fg"], max_depth=MAX_DEPTH,
            seed=1 + int(seed))
        albedo, emission = r.base()
        st["albedo"], st["emission"] = albedo, emission
        # target: what a render with other parameters would average to
        other, _ = perturbed_parameters(albedo, emission, int(seed))
        st["target"] = np.broadcast_to(0.5 * other.mean(axis=0), r.shape).astype(np.float32)
    elif kind == "scene":
        ctx = st["ctx"] = Context(0)
        st["mesh"] = _room_mesh(case["grid"], int(seed))
        st["scene"] = S.Scene(ctx)
        st["rays"] = _camera_rays(case["side"], case["side"], 1, seed)
    else:
        raise ValueError(kind)
    return st


def _room_mesh(grid, seed):
    """The Cornell room over a displaced floor of 2 (grid - 1)^2 triangles."""
    return S.cornell_box(seed) + S.heightfield(grid, 0.05, seed + 1, S.material(rho=S.WHITE), "ground",
                                               amp_max=0.015, wl=(0.08, 0.4))


# -------------------------------------------------------------------- run

def _device_radiance(st, case):
    ctx, q = st["ctx"], st["queries"]
    ctx.check(ctx.lib.pm_photonmap_radiance_device(
        ctx.handle, st["map"].map_id, q.data_ptr(), q.shape[0], case["k"], case["n"],
        st["out"].data_ptr(), torch.cuda.current_stream().cuda_stream),
        "pm_photonmap_radiance_device")
    return st["out"]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "knn":
        idx, count, maxd2 = state["map"].query_knn(state["queries"], case["k"])
        return {"idx": idx, "count": count, "maxdist2": maxd2}
    if kind == "radiance":
        if case["host"]:
            return state["map"].radiance(state["queries"], case["k"], case["n"])
        return _device_radiance(state, case)
    if kind == "rebuild":
        ctx, p = state["ctx"], state["photons"]
        ctx.check(ctx.lib.pm_photonmap_build_device(
            ctx.handle, state["map"].map_id, p.data_ptr(), p.shape[0],
            torch.cuda.current_stream().cuda_stream), "pm_photonmap_build_device")
        return _device_radiance(state, case)
    if kind == "frame":
        stats = state["pmi"].build(state["scene"], seed=1 + state["seed"])
        image, rs = state["pmi"].render(state["camera"], case["width"], case["height"], case["spp"],
                                        n_gather=case["n_gather"])
        return {"image": image, "stored": [v["stored"] for v in stats.values()],
                "samples": rs["samples"], "dropped": rs["dropped_nan"] + rs["dropped_negative"]}
    if kind == "batch":
        b = state["batch"]
        b.render()
        return [b.image(i) for i in range(case["scenes"])]
    if kind == "gradient":
        loss, ga, ge, image = state["renderer"].loss_and_grad(state["albedo"], state["emission"],
                                                              state["target"])
        return {"loss": loss, "albedo": ga, "emission": ge, "image": image}
    sc = state["scene"]
    sc.setMesh(state["mesh"])
    sc.build()
    hits = sc.intersect(*state["rays"])
    return {name: np.ascontiguousarray(hits[name]) for name in hits.dtype.names}


# ------------------------------------------------------------------- work

def _map_size(case):
    return int(case["n"] * (STORED_PER_EMITTED if case["photons"] == "traced" else 1))


def _n_queries(case):
    if case.get("queries") == "camera":
        return int(HITS_PER_RAY * case["side"] ** 2 * case["spp"])
    return case["nq"]


def work(case):
    kind = case["kind"]
    if kind == "knn":  # positions and queries in, index lists out
        return {"bytes": 12 * case["n"] + case["nq"] * (12 + 4 * case["k"] + 8),
                "flops": 8 * case["nq"] * case["k"]}
    if kind in ("radiance", "rebuild"):  # 36-B photons, 48-B queries, RGB out
        n, nq = _map_size(case), _n_queries(case)
        return {"bytes": 36 * n + 60 * nq, "flops": 20 * nq * case["k"]}
    if kind == "scene":  # 72 B of vertices and normals and a 32-B material per face
        faces, rays = 36 + 2 * (case["grid"] - 1) ** 2, case["side"] ** 2
        return {"bytes": 104 * faces + 48 * rays, "flops": 30 * rays * math.log2(faces)}
    if kind == "batch":
        # log-uniform sizes: mean (b - a) / ln(b / a)
        mean = lambda a, b: (b - a) / math.log(max(b, 1.001 * a) / a)  # noqa: E731
        px = mean(128, case["side_max"]) ** 2 * case["scenes"]
        emit = mean(50_000, case["photons_max"]) * case["scenes"]
        faces, k = mean(1_000, case["tri_max"]) * case["scenes"], 75
        samples, maps = px * case["spp"], STORED_PER_EMITTED
    else:
        side2 = case["side"] ** 2 if kind == "gradient" else case["width"] * case["height"]
        px, samples = side2, side2 * case["spp"]
        emit = case["photons"] * (1 + (case.get("mult", 1.0) if case["fg"] else 0))
        faces = 563_238 if case.get("scene") == "caustics" else 36
        maps = 0.5 if case.get("scene") == "caustics" else STORED_PER_EMITTED
        k = case["k"] * (1 + case.get("n_gather", 1) if case["fg"] else 1)
    # geometry read, photon maps written and read, image written; rays of the
    # trace and the camera pass, and the estimates
    rays = emit * (1 + maps) + samples * (2 + (case.get("n_gather", 1) if case.get("fg") else 0))
    flops = 30 * rays * math.log2(faces) + 20 * samples * k
    nbytes = 104 * faces + 72 * maps * emit + 12 * px
    if kind == "gradient":
        flops, nbytes = 2 * flops, 2 * nbytes
    return {"bytes": int(nbytes), "flops": int(flops)}


# ------------------------------------------------------------------ exact

def _exact_knn(pos, q, k):
    """Exact k nearest of q (m, 3) among pos (n, 3) in float64 on the GPU:
    (squared distances, indices), each (m, min(k, n)). Queries are taken cell by
    cell of a coarse grid, each against the photons of a box around the cell;
    the box grows until it holds every k-th distance."""
    n, m = pos.shape[0], q.shape[0]
    k = min(k, n)
    lo = torch.minimum(pos.min(0).values, q.min(0).values)
    ext = (torch.maximum(pos.max(0).values, q.max(0).values) - lo).clamp_min(1e-12)
    grid = int(max(1, min(24, round((n / 4000.0) ** 0.5))))
    cell = lambda x: ((x - lo) / ext * grid).long().clamp_(0, grid - 1)  # noqa: E731
    flat = lambda c: (c[:, 0] * grid + c[:, 1]) * grid + c[:, 2]  # noqa: E731
    porder = torch.argsort(flat(cell(pos)))
    ps = pos[porder]
    pcount = torch.bincount(flat(cell(pos)), minlength=grid ** 3).cpu().numpy()
    pstart = np.concatenate([[0], np.cumsum(pcount)])
    qorder = torch.argsort(flat(cell(q)))
    qcount = torch.bincount(flat(cell(q)), minlength=grid ** 3).cpu().numpy()
    qstart = np.concatenate([[0], np.cumsum(qcount)])
    d2 = torch.empty((m, k), device=pos.device, dtype=torch.float64)
    idx = torch.empty((m, k), device=pos.device, dtype=torch.int64)
    size = (ext / grid)
    for c in np.nonzero(qcount)[0].tolist():
        cx, cy, cz = c // (grid * grid), c // grid % grid, c % grid
        todo = qorder[int(qstart[c]):int(qstart[c + 1])]
        w = 1
        while todo.numel():
            x0, y0, z0 = max(0, cx - w), max(0, cy - w), max(0, cz - w)
            x1, y1, z1 = (min(grid - 1, v + w) for v in (cx, cy, cz))
            rows = [slice(int(pstart[(x * grid + y) * grid + z0]),
                          int(pstart[(x * grid + y) * grid + z1 + 1]))
                    for x in range(x0, x1 + 1) for y in range(y0, y1 + 1)]
            rows = [r for r in rows if r.stop > r.start]
            whole = (x0, y0, z0) == (0, 0, 0) and (x1, y1, z1) == (grid - 1,) * 3
            have = sum(r.stop - r.start for r in rows)
            if have < k:
                w *= 2
                continue
            cand = torch.cat([ps[r] for r in rows])
            cid = torch.cat([porder[r] for r in rows])
            left = []
            step = max(1, 40_000_000 // have)
            # distance from a query to the faces of the box that are inside the grid
            blo = lo + size * torch.tensor([x0, y0, z0], device=pos.device)
            bhi = lo + size * torch.tensor([x1 + 1, y1 + 1, z1 + 1], device=pos.device)
            open_lo = torch.tensor([x0 > 0, y0 > 0, z0 > 0], device=pos.device)
            open_hi = torch.tensor([v < grid - 1 for v in (x1, y1, z1)], device=pos.device)
            for part in todo.split(step):
                t = q[part]
                e = sum((t[:, a, None] - cand[None, :, a]) ** 2 for a in range(3))
                near, at = torch.topk(e, k, dim=1, largest=False, sorted=True)
                inf = torch.full_like(t, math.inf)
                room = torch.minimum(torch.where(open_lo, t - blo, inf),
                                     torch.where(open_hi, bhi - t, inf)).min(1).values
                ok = torch.ones_like(room, dtype=torch.bool) if whole else (
                    (room > 0) & (near[:, -1] <= (room * (1 - 1e-12)) ** 2))
                d2[part[ok]], idx[part[ok]] = near[ok], cid[at[ok]]
                left.append(part[~ok])
            todo = torch.cat(left)
            w *= 2
    return d2, idx


def _exact_radiance(photons, queries, k, n_emitted):
    """computeRadianceWithPhotonMap with the Lambert BRDF in float64."""
    p, q = photons.double(), queries.double()
    d2, idx = _exact_knn(p[:, 3:6].contiguous(), q[:, 0:3].contiguous(), k)
    rho = q[:, [3, 7, 11]]
    out = torch.empty((q.shape[0], 3), device=q.device, dtype=torch.float64)
    for a in range(0, q.shape[0], 65_536):
        b = min(a + 65_536, q.shape[0])
        near = p[idx[a:b]]
        ns = q[a:b, 8:11]
        seen = ((near[..., 6:9] * ns[:, None]).sum(-1) >= 0) & (
            (q[a:b, 4:7] * ns).sum(-1) >= 0)[:, None]
        total = (near[..., 0:3] * seen[..., None]).sum(1)
        out[a:b] = rho[a:b] / math.pi * total / (n_emitted * math.pi * d2[a:b, -1:])
    return out


def _exact_hits(mesh, o, d):
    """Closest hits by the ray/triangle equations in float64."""
    v = torch.from_numpy(np.asarray(mesh.vertices, np.float32)).cuda().double().reshape(-1, 3, 3)
    p0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    ng = torch.linalg.cross(e1, e2)
    O, D = (torch.from_numpy(x).cuda().double() for x in (o, d))
    res = torch.zeros((O.shape[0], 3), device="cuda", dtype=torch.float64)
    step = max(1, 30_000_000 // v.shape[0])
    for a in range(0, O.shape[0], step):
        oo, dd = O[a:a + step, None], D[a:a + step, None]
        det = -(dd * ng).sum(-1)
        s = oo - p0
        t = (s * ng).sum(-1) / det
        sd = torch.linalg.cross(s, dd.expand_as(s))
        u, w = (sd * e2).sum(-1) / det, -(sd * e1).sum(-1) / det
        ok = (det != 0) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t >= 1e-5)
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, at = t.min(1)
        hit = torch.isfinite(best)
        got = torch.stack([best, u.gather(1, at[:, None])[:, 0], w.gather(1, at[:, None])[:, 0]], 1)
        res[a:a + step] = torch.where(hit[:, None], got, torch.zeros_like(got))
    return res


def exact(case, seed):
    """What run() returns, in 64 bits. None where no such value exists:
    indices and counts, and everything that follows random paths (frames,
    batches, gradients: which way a path goes hangs on the 32-bit rounding of
    each step, so a 64-bit run follows other paths)."""
    kind = case["kind"]
    if kind == "knn":
        p = _photons(case["photons"], case["n"], seed)[:, 3:6].double().contiguous()
        q = _wall_queries(case["nq"], seed)[:, :3].double().contiguous()
        d2, _ = _exact_knn(p, q, case["k"])
        return {"idx": None, "count": None, "maxdist2": d2[:, -1]}
    if kind in ("radiance", "rebuild") and case["photons"] != "traced":
        photons, queries = _photons(case["photons"], case["n"], seed), None
        if case["queries"] == "walls":
            queries = _wall_queries(case["nq"], seed)
            return _exact_radiance(photons, queries, case["k"], case["n"])
        return None
    if kind == "radiance":
        # the photons and the hit points are the inputs here, read back
        st = prepare(dict(case, host=False), seed)
        photons = torch.from_numpy(st["map"].photons()).cuda()
        return _exact_radiance(photons, st["queries"], case["k"], case["n"])
    if kind == "scene" and case["side"] ** 2 * case["grid"] ** 2 <= 1e10:
        st_rays = _camera_rays(case["side"], case["side"], 1, seed)
        r = _exact_hits(_room_mesh(case["grid"], int(seed)), *st_rays)
        return {"t": r[:, 0], "u": r[:, 1], "v": r[:, 2], "prim": None}
    return None
