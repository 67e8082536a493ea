"""Timed workloads over the library's public entry points.

Each case is one call sequence of a program that uses the library: build a
BVH over triangles and trace an image, trace explicit rays against a kept
BVH, run a kept batch of meshes, or the reference's own host calls
(Builder.build_hierarchy + trace).  Inputs are made on the GPU from a seed,
in the shapes and sizes of sequoia_gb300/scenes.py: displaced icospheres,
Gaussian triangle soups and height-field terrains.

kinds
  frame    build over device triangles, then one camera image (hits and
           heatmap, or the heatmap alone for the packet and bundle tracers)
           into device buffers
  rays     explicit rays in one device buffer against a kept BVH
  batches  explicit rays in many device buffers, one launch
  meshes   a kept batch: every mesh built and its image traced, one graph
  image    host triangles through the reference's host interface: build,
           node array on the host, heatmap bytes on the host
"""
import math

import numpy as np
import torch

import sequoia_gb300 as sq
from sequoia_gb300 import scenes

_state = {}
FLT_MAX = 3.4028234663852886e38


def _context():
    """One context for the program, on the stream that torch works on."""
    if "ctx" not in _state:
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        torch.cuda.set_stream(stream)
        _state["ctx"] = sq.Context(torch.cuda.current_device(), stream=stream.cuda_stream)
    return _state["ctx"]


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # a preview of a small mesh: launches and latency are all of it
        dict(name="preview_1k", kind="frame", scene="icosphere", tris=1280, builder="morton", wide=True,
             mode="closest", camera="pinhole", width=64, height=48),
        # the small benchmark configuration: one object, a quality build, a full image
        dict(name="object_sah16_1080p", kind="frame", scene="icosphere", tris=81920, builder="sah", bins=16, leaf=4,
             wide=True, mode="closest", camera="pinhole", width=1920, height=1080),
        # the headline configuration: a rebuilt scene and a 4K image each frame
        dict(name="soup2m_morton_4k", kind="frame", scene="soup", tris=2000000, builder="morton", wide=True,
             mode="closest", camera="pinhole", width=3840, height=2160),
        # a terrain: every triangle small, most rays hit
        dict(name="terrain4m_morton_1080p", kind="frame", scene="terrain", tris=4194304, builder="morton", wide=True,
             mode="closest", camera="pinhole", width=1920, height=1080),
        # the reference's default: its SAH builder and its tracer, on the device
        dict(name="soup2m_sah8_ref_1080p", kind="frame", scene="soup", tris=2000000, builder="sah", bins=8, leaf=8,
             wide=False, mode="ref", camera="reference", width=1920, height=1080),
        # the reference's grid builder and packet tracer, a ragged mesh
        dict(name="soup300k_grid_packet8", kind="frame", scene="soup", tris=300007, builder="grid", bins=8, leaf=8,
             wide=False, mode="packet", k=8, camera="reference", width=1280, height=720),
        # one diffuse bounce from the terrain's surface (the second half of the terrain configuration)
        dict(name="terrain4m_bounce", kind="rays", scene="terrain", tris=4194304, builder="morton", wide=True,
             mode="closest", order="surface", rays=567775),
        # ambient occlusion on the plain FP32 tree: any hit, per-lane schedule, odd sizes
        dict(name="soup500k_anyhit_binary", kind="rays", scene="soup", tris=500009, builder="morton", wide=False,
             mode="anyhit", sched="refill", order="random", rays=1000003),
        # the stress configuration: incoherent rays of many callers against a large scene
        dict(name="soup8m_incoherent_16m", kind="batches", scene="soup", tris=8000000, builder="morton", wide=True,
             mode="closest", rays=1 << 24, batches=64),
        # the many-meshes configuration with either batch builder
        dict(name="meshes256_morton", kind="meshes", meshes=256, lo=1000, hi=200000, side_lo=64, side_hi=512,
             builder="morton", wide=True, mode="closest"),
        dict(name="meshes64_sah16", kind="meshes", meshes=64, lo=1000, hi=200000, side_lo=64, side_hi=512,
             builder="sah", bins=16, leaf=4, wide=True, mode="closest"),
        # the reference's published run: a 69,451-triangle object through its host interface
        dict(name="host_object_69k", kind="image", scene="icosphere", tris=69451, builder="sah", width=1920,
             height=1080),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scene(rng, most):
    scene = rng.choice(["icosphere", "soup", "terrain"])
    n = _log_int(rng, 1000, min(most, 320000) if scene == "icosphere" else most)
    if scene == "terrain":
        n = 2 * max(4, int(round(math.sqrt(n / 4)))) * (2 * max(4, int(round(math.sqrt(n / 4)))))
    return scene, n


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "rays", "rays", "batches", "meshes", "image"])
    if kind == "frame":
        scene, n = _scene(rng, 4000000)
        c = dict(kind=kind, scene=scene, tris=n)
        c["builder"] = rng.choice(["morton", "morton", "morton60", "sah", "grid"])
        if c["builder"] in ("sah", "grid"):
            c.update(bins=rng.choice([8, 16, 32]), leaf=rng.choice([4, 8]))
        c["mode"] = rng.choice(["closest", "closest", "closest", "anyhit", "ref", "packet", "bundle"])
        if c["mode"] in ("packet", "bundle"):
            c["k"] = rng.choice([4, 8]) if c["mode"] == "packet" else rng.choice([16, 64])
        c["wide"] = c["mode"] in ("closest", "anyhit") and rng.random() < 0.75
        coherent = c["mode"] in ("packet", "bundle", "ref")
        c["camera"] = "reference" if coherent else "pinhole"
        c["width"] = _log_int(rng, 64, 1920 if coherent else 3840)
        c["height"] = max(48, int(c["width"] * rng.uniform(0.5, 0.75)))
        if coherent:  # whole packet blocks
            c["width"], c["height"] = c["width"] // 16 * 16, c["height"] // 16 * 16
        return c
    if kind == "rays":
        scene, n = _scene(rng, 4000000)
        return dict(kind=kind, scene=scene, tris=n, builder=rng.choice(["morton", "sah"]), bins=8, leaf=8,
                    wide=rng.random() < 0.75, mode=rng.choice(["closest", "anyhit"]),
                    order=rng.choice(["surface", "random"]), rays=_log_int(rng, 1000, 2000000))
    if kind == "batches":
        scene, n = _scene(rng, 4000000)
        return dict(kind=kind, scene=scene, tris=n, builder="morton", wide=rng.random() < 0.75,
                    mode=rng.choice(["closest", "anyhit"]), rays=_log_int(rng, 20000, 4000000),
                    batches=_log_int(rng, 2, 64))
    if kind == "meshes":
        hi = _log_int(rng, 3000, 200000)
        c = dict(kind=kind, meshes=_log_int(rng, 4, 200), lo=1000, hi=hi, side_lo=64, side_hi=_log_int(rng, 96, 512),
                 builder=rng.choice(["morton", "sah"]), wide=rng.random() < 0.5, mode=rng.choice(["closest", "anyhit"]))
        if c["builder"] == "sah":
            c.update(bins=rng.choice([8, 16, 32]), leaf=rng.choice([4, 8]))
        return c
    scene, n = _scene(rng, 150000)
    w = _log_int(rng, 320, 1920) // 16 * 16
    return dict(kind=kind, scene=scene, tris=n, builder=rng.choice(["morton", "sah", "grid"]), width=w,
                height=w // 2 // 16 * 16)


# ------------------------------------------------------- scenes, on the device

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _base_icosphere(level):
    """Vertices and faces of an undisplaced icosphere (they do not depend on the seed)."""
    key = ("ico", level)
    if key not in _state:
        v, f = scenes.icosphere(level)
        _state[key] = (torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda())
    return _state[key]


def _icosphere(n, seed):
    """The first n triangles of the smallest displaced icosphere with at least n."""
    level = 0
    while 20 * 4 ** level < n:
        level += 1
    v, f = _base_icosphere(level)
    g = _generator(seed)
    abc = _uniform(g, 1.0, 4.0, 4, 3)
    phi = _uniform(g, 0.0, 2.0 * math.pi, 4)
    r = 1.0 + 0.05 * torch.sin(v @ abc.T + phi).sum(1)
    return (v * r[:, None]).float()[f[:n]].reshape(n, 9).contiguous()


def _soup(n, clusters, seed):
    """Equilateral triangles of lognormal edge length around Gaussian clusters in [-10, 10]^3."""
    g = _generator(seed)
    centres = _uniform(g, -10.0, 10.0, clusters, 3).float()
    sigma = _uniform(g, 0.2, 2.0, clusters).float()
    out = torch.empty(n, 9, device="cuda")
    ang = torch.arange(3, device="cuda") * (2.0 * math.pi / 3.0)
    ca, sa = ang.cos()[None, :, None], ang.sin()[None, :, None]
    for s in range(0, n, 1 << 22):
        m = min(1 << 22, n - s)
        comp = torch.randint(0, clusters, (m,), generator=g, device="cuda")
        c = centres[comp] + sigma[comp, None] * torch.randn(m, 3, generator=g, device="cuda")
        size = torch.exp(torch.randn(m, generator=g, device="cuda") * 0.5 + math.log(0.02)) / math.sqrt(3.0)
        e1 = torch.randn(m, 3, generator=g, device="cuda")
        e1 = e1 / e1.norm(dim=1, keepdim=True)
        e2 = torch.linalg.cross(e1, torch.randn(m, 3, generator=g, device="cuda"))
        e2 = e2 / e2.norm(dim=1, keepdim=True)
        v = c[:, None, :] + size[:, None, None] * (ca * e1[:, None, :] + sa * e2[:, None, :])
        out[s:s + m] = v.reshape(m, 9)
    return out


def _terrain(n, seed):
    """nx x nz quads (nx = 2 nz), two triangles each, over [-1, 1] x [-0.5, 0.5]; 8 octaves of value noise."""
    nz = int(round(math.sqrt(n / 4)))
    nx = n // 2 // nz
    g = _generator(seed)
    x = torch.linspace(-1.0, 1.0, nx + 1, device="cuda", dtype=torch.float64)[None, :].expand(nz + 1, nx + 1)
    z = torch.linspace(-0.5, 0.5, nz + 1, device="cuda", dtype=torch.float64)[:, None].expand(nz + 1, nx + 1)
    y, norm = torch.zeros_like(x), 0.0
    for o in range(8):
        freq = 4 << o
        lat = _uniform(g, -1.0, 1.0, freq + 2, 2 * freq + 2)
        gx, gz = (x + 1.0) * freq, (z + 0.5) * freq
        ix, iz = gx.floor().long().clamp(0, 2 * freq), gz.floor().long().clamp(0, freq)
        fx, fz = gx - ix, gz - iz
        sx, sz = fx * fx * (3 - 2 * fx), fz * fz * (3 - 2 * fz)
        v0 = lat[iz, ix] + (lat[iz, ix + 1] - lat[iz, ix]) * sx
        v1 = lat[iz + 1, ix] + (lat[iz + 1, ix + 1] - lat[iz + 1, ix]) * sx
        y += 0.5 ** o * (v0 + (v1 - v0) * sz)
        norm += 0.5 ** o
    v = torch.stack([x, 0.2 * y / norm, z], -1).float()
    a, b, c, d = v[:-1, :-1], v[:-1, 1:], v[1:, 1:], v[1:, :-1]
    return torch.stack([torch.cat([a, b, c], -1), torch.cat([a, c, d], -1)], 2).reshape(-1, 9).contiguous()


def _triangles(case, seed):
    if case["scene"] == "icosphere":
        return _icosphere(case["tris"], seed)
    if case["scene"] == "terrain":
        return _terrain(case["tris"], seed)
    return _soup(case["tris"], 256 if case["tris"] > 4000000 else 64, seed)


def _camera(case, tris):
    """The configurations' cameras; the reference camera stands as far in front of the scene as the benchmark's."""
    if case["camera"] == "reference":
        v = tris.view(-1, 3)
        lo, hi = v.amin(0).tolist(), v.amax(0).tolist()
        c = [(a + b) * 0.5 for a, b in zip(lo, hi)]
        return dict(camera="reference", width=case["width"], height=case["height"],
                    origin=(c[0], c[1], 2.0 * lo[2] - c[2]))
    eye = {"icosphere": (0.0, 0.0, 3.0), "soup": (0.0, 0.0, -40.0), "terrain": (0.0, 0.6, -1.2)}[case["scene"]]
    return dict(camera="pinhole", width=case["width"], height=case["height"], origin=eye, target=(0.0, 0.0, 0.0),
                up=(0.0, 1.0, 0.0), vfov=60.0)


def _ray_buffer(case, tris, count, seed):
    """(count, 8) float32 {origin, tmin, direction, tmax}: random through the scene box, or one
    cosine-weighted bounce from points spread evenly over the triangle list."""
    g = _generator(seed + 77)
    d = torch.randn(count, 3, generator=g, device="cuda")
    d = d / d.norm(dim=1, keepdim=True)
    r = torch.empty(count, 8, device="cuda")
    if case.get("order") == "surface":
        at = (torch.arange(count, device="cuda", dtype=torch.int64) * len(tris)) // count
        t = tris[at].view(count, 3, 3)
        w = torch.rand(count, 2, generator=g, device="cuda")
        w = torch.where((w.sum(1) > 1)[:, None], 1 - w, w)
        p = t[:, 0] + w[:, :1] * (t[:, 1] - t[:, 0]) + w[:, 1:] * (t[:, 2] - t[:, 0])
        nrm = torch.linalg.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
        nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
        nrm = torch.where((nrm[:, 1] < 0)[:, None], -nrm, nrm)
        d = nrm + 0.999 * d
        d = d / d.norm(dim=1, keepdim=True)
        r[:, 0:3] = p + 1e-4 * nrm
    else:
        v = tris.view(-1, 3)
        lo, hi = v.amin(0), v.amax(0)
        r[:, 0:3] = lo + (hi - lo) * torch.rand(count, 3, generator=g, device="cuda")
    r[:, 3] = 0.0
    r[:, 4:7] = d
    r[:, 7] = 3.4e38
    return r


def _mesh_list(case, seed):
    """Meshes of log-uniform sizes, icospheres and soups, each with a square image of log-uniform side."""
    rng = np.random.default_rng(4000)  # sizes are the case's; the shapes in them are the seed's
    meshes = []
    for i in range(case["meshes"]):
        n = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        side = int(round(math.exp(rng.uniform(math.log(case["side_lo"]), math.log(case["side_hi"])))))
        t = _icosphere(n, seed * 1000 + i) if rng.uniform() < 0.5 else _soup(n, 8, seed * 1000 + i)
        meshes.append((t, side))
    box = torch.stack([torch.stack([t.view(-1, 3).amin(0), t.view(-1, 3).amax(0)]) for t, _ in meshes]).tolist()
    out = []
    for (t, side), (lo, hi) in zip(meshes, box):
        c = [(a + b) * 0.5 for a, b in zip(lo, hi)]
        ext = max(b - a for a, b in zip(lo, hi))
        out.append(dict(tris=t, camera="pinhole", width=side, height=side,
                        origin=(c[0], c[1] + 0.5 * ext, c[2] - 2.5 * ext), target=tuple(c), up=(0.0, 1.0, 0.0),
                        vfov=50.0))
    return out


# ------------------------------------------------------------ prepare and run

def _build(ctx, case, tris):
    kw = dict(wide=case["wide"])
    if case["builder"] == "morton60":
        kw.update(builder="morton", morton64=True)
    elif case["builder"] == "morton":
        kw.update(builder="morton")
    else:
        kw.update(builder=case["builder"], bins=case["bins"], leaf=case["leaf"])
    return ctx.build(tris, **kw)


def _out_buffers(rays, hits=True, heat=True):
    return (torch.empty(rays, 3, dtype=torch.int32, device="cuda") if hits else False,
            torch.empty(rays * 3, dtype=torch.uint8, device="cuda") if heat else False)


def prepare(case, seed):
    ctx = _context()
    s = dict(case=case, ctx=ctx)
    kind = case["kind"]
    if kind == "meshes":
        meshes = _mesh_list(case, seed)
        rays = sum(m["width"] * m["height"] for m in meshes)
        s["hits"], s["heat"] = _out_buffers(rays)
        kw = dict(builder="sah", bins=case["bins"], leaf=case["leaf"]) if case["builder"] == "sah" else {}
        s["batch"] = ctx.batch(meshes, mode=case["mode"], wide=case["wide"], **kw)
        return s
    tris = _triangles(case, seed)
    if kind == "image":
        s["tris"] = tris.cpu().numpy()
        lo, hi = s["tris"].reshape(-1, 3).min(0), s["tris"].reshape(-1, 3).max(0)
        c = (lo + hi) * np.float32(0.5)
        s["origin"] = (float(c[0]), float(c[1]), float(2 * lo[2] - c[2]))
        return s
    s["tris"] = tris
    if kind == "frame":
        s["camera"] = _camera(case, tris)
        coherent = case["mode"] in ("packet", "bundle")
        s["hits"], s["heat"] = _out_buffers(case["width"] * case["height"], hits=not coherent)
        return s
    s["bvh"] = _build(ctx, case, tris)
    rays = _ray_buffer(case, tris, case["rays"], seed)
    s["hits"], s["heat"] = _out_buffers(case["rays"], heat=False)
    if kind == "batches":
        sizes = scenes.batch_sizes(case["rays"], case["batches"], lo=max(1, case["rays"] // case["batches"] // 8),
                                   hi=max(2, case["rays"] // case["batches"] * 8), seed=5)
        cuts = np.concatenate([[0], np.cumsum(sizes)])
        s["rays"] = [rays[cuts[k]:cuts[k + 1]].clone() for k in range(len(sizes))]
    else:
        s["rays"] = rays
    return s


def _outputs(s):
    out = {}
    if s["hits"] is not False:
        out.update(id=s["hits"][:, 0], t=s["hits"].view(torch.float32)[:, 1], tests=s["hits"][:, 2])
    if s["heat"] is not False:
        out["heat"] = s["heat"]
    return out


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "frame":
        bvh = _build(ctx, case, s["tris"])
        ctx.trace(bvh, case["mode"], k=case.get("k", 0), hits=s["hits"], heatmap=s["heat"], **s["camera"])
        bvh.free()
    elif kind == "rays":
        ctx.trace(s["bvh"], case["mode"], rays=s["rays"], hits=s["hits"], sched=case.get("sched"))
    elif kind == "batches":
        ctx.trace_batches(s["bvh"], case["mode"], s["rays"], hits=s["hits"])
    elif kind == "meshes":
        s["batch"].run(hits=s["hits"], heatmap=s["heat"])
    else:
        make = {"sah": sq.Builder.build_hierarchy, "morton": sq.Builder.build_hierarchy_morton,
                "grid": sq.Builder.build_hierarchy_grid}[case["builder"]]
        h = make(s["tris"])
        return {"heat": sq.trace(h, case["width"], case["height"], s["origin"]), "nodes": h.node_count}
    return _outputs(s)


# ------------------------------------------------- what a pass cannot do without

def _mesh_totals(case):
    rng = np.random.default_rng(4000)
    tris = rays = 0
    for _ in range(case["meshes"]):
        tris += int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        rays += int(round(math.exp(rng.uniform(math.log(case["side_lo"]), math.log(case["side_hi"]))))) ** 2
        rng.uniform()
    return tris, rays


def work(case):
    """Triangles (36 B) in, explicit rays (32 B) in, a hit record (12 B) and a pixel (3 B) out per ray, and the
    node array (3 n records of 32 B) where the call returns it; a box and centroid per triangle and one slab
    test per ray."""
    kind = case["kind"]
    if kind == "meshes":
        tris, rays = _mesh_totals(case)
        return dict(bytes=36 * tris + 15 * rays, flops=30 * tris + 25 * rays)
    if kind in ("rays", "batches"):
        return dict(bytes=44 * case["rays"], flops=25 * case["rays"])
    rays = case["width"] * case["height"]
    per_ray = 3 if kind == "image" or case["mode"] in ("packet", "bundle") else 15
    nodes = 96 * case["tris"] if kind == "image" else 0
    return dict(bytes=36 * case["tris"] + nodes + per_ray * rays, flops=30 * case["tris"] + 25 * rays)


# --------------------------------------------------- 64-bit distances, small cases

def _camera_rays64(cam):
    w, h = cam["width"], cam["height"]
    eye = torch.tensor(cam["origin"], dtype=torch.float64, device="cuda")
    f = torch.tensor(cam["target"], dtype=torch.float64, device="cuda") - eye
    f = f / f.norm()
    r = torch.linalg.cross(f, torch.tensor(cam["up"], dtype=torch.float64, device="cuda"))
    r = r / r.norm()
    u = torch.linalg.cross(r, f)
    th = math.tan(cam["vfov"] * math.pi / 360.0)
    px = ((torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w * 2 - 1) * (th * w / h)
    py = ((torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h * 2 - 1) * th
    py, px = torch.meshgrid(py, px, indexing="ij")
    d = f + px.reshape(-1, 1) * r + py.reshape(-1, 1) * u
    d = d / d.norm(dim=1, keepdim=True)
    return eye.expand_as(d), d


def _closest64(tris, o, d):
    """Nearest hit distance of each ray (0 where none), every ray against every triangle."""
    t = tris.double().view(-1, 3, 3)
    v0, e1, e2 = t[:, 0], t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]
    out = torch.zeros(len(o), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 23) // len(t))
    for a in range(0, len(o), step):
        oo, dd = o[a:a + step, None, :], d[a:a + step, None, :]
        p = torch.linalg.cross(dd.expand(-1, len(t), -1), e2[None].expand(len(oo), -1, -1))
        det = (p * e1).sum(-1)
        s = oo - v0
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand(len(oo), -1, -1))
        v = (q * dd).sum(-1) / det
        k = (q * e2).sum(-1) / det
        ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (k >= 0)
        k = torch.where(ok, k, torch.inf).amin(1)
        out[a:a + step] = torch.where(torch.isfinite(k), k, 0.0)
    return out


def exact(case, seed):
    """The hit distances in 64 bits where every ray can be tested against every triangle; ids, counts and
    heatmap bytes are whole numbers."""
    if case["kind"] not in ("frame", "rays") or case["mode"] != "closest":
        return None
    rays = case["rays"] if case["kind"] == "rays" else case["width"] * case["height"]
    if rays * case["tris"] > 8e9:
        return None
    tris = _triangles(case, seed)
    if case["kind"] == "frame":
        t = _closest64(tris, *_camera_rays64(_camera(case, tris)))
        return dict(id=None, t=t, tests=None, heat=None)
    r = _ray_buffer(case, tris, case["rays"], seed).double()
    return dict(id=None, t=_closest64(tris, r[:, 0:3], r[:, 4:7]), tests=None)
