"""Performance cases of the framework's public entry points (renzoku_b200/rzk.py).

Each case is one call (or the two calls that belong together) that a program using this
framework makes, at sizes from the repository's own configurations, tests and benchmark:

  gather      VirtualPointLightCuda.gather: one frame of the many-light integrator
  batch       GatherBatch.run: a queue of small frames in one launch
  fill        VirtualPointLightCuda.fill / incident_radiance: the light transport matrix
  cluster     ClusterBuilderCuda.alphas + cluster_by_sampling on such a matrix
  segments    AggregateCuda.hit_segments: visibility between point pairs
  rays        AggregateCuda.hit_rays: closest hits of scattered rays
  spawn       VplGeneratorCuda.spawn: tracing the VPLs of a frame
  lightslice  LightSliceCuda.gather: one frame of the clustered gather
  guided      LightSliceCuda.guided_render: one frame of guided path tracing
  rebuild     AggregateCuda.rebuild, then the first queries on the new trees

Scenes are the procedural rooms of renzoku_b200/scenegen.py: "room" (36 triangles, boxes),
"objects" (boxes and spheres of Lambertian, Phong and Ward materials, about 150 triangles
each) and "spheres" (48 triangles each, Lambertian).
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from renzoku_b200 import instances, rzk
from renzoku_b200 import scenegen as sg

RECORD = 96   # bytes of a receiver or VPL record
MODES = {"none": rzk.CLAMP_NONE, "form_factor": rzk.CLAMP_FORM_FACTOR,
         "reflectivity": rzk.CLAMP_REFLECTIVITY, "radiance": rzk.CLAMP_RADIANCE}
TAUS = {"none": 0.0, "form_factor": 1.0, "reflectivity": 0.05, "radiance": 0.05}
BRUTE = 2e10  # most (ray, triangle) tests an exact answer is worked out with


def listed():
    return [
        # the smallest frame: a thumbnail or one tile, where launches and latency count
        {"name": "gather_small", "kind": "gather", "scene": "room", "count": 0, "width": 61, "height": 47,
         "n_vpl": 333, "clamp": "form_factor", "tiled": True},
        # the box room at its own size: few triangles, most pairs visible
        {"name": "gather_room", "kind": "gather", "scene": "room", "count": 0, "width": 256, "height": 256,
         "n_vpl": 4096, "clamp": "radiance", "tiled": True},
        # the headline frame: 300k triangles, mixed materials
        {"name": "gather_scaled", "kind": "gather", "scene": "objects", "count": 2000, "width": 512, "height": 512,
         "n_vpl": 32768, "clamp": "radiance", "tiled": True},
        # a queue of small requests of different scenes, sizes and VPL counts in one launch
        {"name": "batch_small", "kind": "batch", "jobs": 10, "sizes": 2025, "tris": 30000, "side": 192, "n_vpl": 3000},
        # the reduced matrix of a row-column sampled image, with its visibility
        {"name": "fill_reduced", "kind": "fill", "scene": "objects", "count": 2000, "width": 20, "height": 13,
         "n_vpl": 10007, "clamp": "radiance", "what": "radiance"},
        # clustering of such a matrix
        {"name": "cluster_10k", "kind": "cluster", "scene": "objects", "count": 400, "width": 16, "height": 16,
         "n_vpl": 10000, "clusters": 300},
        # visibility queries between shading points and VPLs
        {"name": "segments_1m", "kind": "segments", "scene": "objects", "count": 2000, "n": 1000003, "n_vpl": 4096},
        # closest hits of rays scattered from surfaces
        {"name": "rays_512k", "kind": "rays", "scene": "objects", "count": 2000, "n": 524288},
        # the VPLs of the headline frame
        {"name": "spawn_24k", "kind": "spawn", "scene": "objects", "count": 2000, "particles": 24000, "bounces": 3},
        # the clustered gather of the headline frame
        {"name": "lightslice_scaled", "kind": "lightslice", "scene": "objects", "count": 2000, "width": 512,
         "height": 512, "n_vpl": 32768, "clamp": "form_factor", "slice": 1024, "clusters": 1000, "slice_clusters": 2000},
        # a guided frame over small spheres
        {"name": "guided_384", "kind": "guided", "scene": "spheres", "count": 6000, "width": 384, "height": 384,
         "n_vpl": 20000, "spp": 4, "bounces": 8, "sampler": "jensen", "slice": 4096, "clusters": 1000},
        # an edited scene: both trees again, then its primary hits and some visibility
        {"name": "rebuild_300k", "kind": "rebuild", "scene": "objects", "count": 2000, "width": 256, "height": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("gather", "gather", "gather", "batch", "fill", "cluster", "segments", "rays", "spawn",
                       "lightslice", "guided", "rebuild"))
    c = {"kind": kind}
    if kind == "batch":
        c.update(jobs=rng.randint(3, 10), sizes=rng.randrange(1 << 20), tris=_log(rng, 10000, 30000),
                 side=_log(rng, 96, 192), n_vpl=_log(rng, 1000, 3000))
        return c
    if kind == "guided":
        side = _log(rng, 96, 384)
        c.update(scene="spheres", count=_log(rng, 200, 6000), width=side, height=max(64, side - rng.randint(0, 31)),
                 n_vpl=_log(rng, 3000, 20000), spp=rng.randint(1, 4), bounces=rng.randint(2, 8),
                 sampler=rng.choice(("jensen", "metropolis")), slice=1024, clusters=_log(rng, 100, 1000))
        return c
    c["scene"] = "objects" if rng.random() < 0.8 else ("spheres" if kind in ("segments", "rays", "rebuild") else "room")
    c["count"] = {"objects": _log(rng, 20, 2000), "spheres": _log(rng, 60, 6000), "room": 0}[c["scene"]]
    if kind == "gather":
        w = _log(rng, 40, 512)
        c.update(width=w, height=_log(rng, 32, min(2 * w, 512)), n_vpl=_log(rng, 200, 32768),
                 clamp=rng.choice(tuple(MODES)), tiled=rng.random() < 0.75)
    elif kind == "fill":
        c.update(width=rng.randint(6, 20), height=rng.randint(4, 13), n_vpl=_log(rng, 500, 10007),
                 clamp=rng.choice(tuple(MODES)), what=rng.choice(("radiance", "radiance", "incident")))
    elif kind == "cluster":
        n = _log(rng, 1000, 10000)
        c.update(width=rng.randint(8, 16), height=rng.randint(8, 16), n_vpl=n, clusters=max(16, n * 3 // 100))
        c.update(scene="objects", count=max(20, min(400, c["count"])))
    elif kind == "segments":
        c.update(n=_log(rng, 5000, 1000003), n_vpl=_log(rng, 200, 4096))
    elif kind == "rays":
        c.update(n=_log(rng, 5000, 524288))
    elif kind == "spawn":
        c.update(particles=_log(rng, 300, 24000), bounces=rng.randint(2, 6))
        c["particles"] = min(c["particles"], 24000 * 3 // c["bounces"])
    elif kind == "lightslice":
        w = _log(rng, 96, 512)
        c.update(scene="objects", count=max(100, c["count"]), width=w, height=max(64, w - rng.randint(0, 63)),
                 n_vpl=_log(rng, 3000, 32768), clamp=rng.choice(tuple(MODES)), slice=1024, clusters=_log(rng, 100, 1000),
                 slice_clusters=_log(rng, 200, 2000))
    else:
        c.update(width=rng.randint(64, 256), height=rng.randint(64, 256))
    return c


# ------------------------------------------------------------------------------- inputs

_CONTEXT = []


def _context():
    if not _CONTEXT:   # one context for the program's life, as a renderer keeps it
        _CONTEXT.append(rzk.Context(0))
    return _CONTEXT[0]


def _scene(case, seed):
    w, h = case.get("width", 256), case.get("height", 256)
    if case["scene"] == "room":
        return sg.room_boxes(w, h)
    if case["scene"] == "spheres":
        return sg.room_spheres(case["count"], w, h, seed=seed)
    return sg.room_objects(case["count"], w, h, seed_geo=seed, seed_mat=seed + 1)


@dataclasses.dataclass
class State:
    case: dict
    scene: sg.Scene
    agg: rzk.AggregateCuda
    seed: int
    cam: rzk.Camera = None
    recv: torch.Tensor = None
    n_recv: int = 0
    vpls: torch.Tensor = None
    scale: float = 1.0
    ev: rzk.VirtualPointLightCuda = None
    a: torch.Tensor = None
    b: torch.Tensor = None
    builder: rzk.ClusterBuilderCuda = None
    ls: rzk.LightSliceCuda = None


def _floats(records):
    return records.view(torch.float32).reshape(-1, RECORD // 4)


def _ints(records):
    return records.view(torch.int32).reshape(-1, RECORD // 4)


def _surface_points(s, n, gen):
    """n shading points of the scene's own image (position and shading normal), drawn with repetition."""
    spec = dataclasses.replace(s.scene.camera, width=256, height=256)
    recv = s.agg.primary(rzk.Camera(spec))
    rows = torch.nonzero(_ints(recv)[:, 21] >= 0)[:, 0]
    rows = rows[torch.randint(rows.numel(), (n,), generator=gen, device="cuda")]
    f = _floats(recv)[rows]
    return f[:, 0:3].contiguous(), f[:, 6:9].contiguous()


def _prepare_batch(case, seed):
    jobs, keep = [], []
    specs = instances.batch_specs(case["jobs"], case["sizes"], tris=(case["tris"] // 3, case["tris"]),
                                  side=(case["side"] // 3, case["side"]), vpls=(case["n_vpl"] // 3, case["n_vpl"]))
    for k, spec in enumerate(specs):
        sc = sg.room_filled(spec.n_tris, spec.width, spec.height, seed + 2 * k)
        agg = rzk.AggregateCuda(_context(), sc)
        recv = agg.primary(rzk.Camera(sc.camera))
        vpls, emitted = instances.spawn_vpls(agg, seed + k, spec.n_vpl)
        n = spec.width * spec.height
        out = torch.zeros((n, 3), dtype=torch.float32, device="cuda")
        jobs.append((agg, recv, n, spec.width, vpls, spec.n_vpl, MODES["radiance"], TAUS["radiance"], 1.0 / emitted, out))
        keep.append((agg, recv, vpls, out))
    return {"case": case, "keep": keep, "batch": rzk.GatherBatch(_context(), rzk.make_jobs(jobs))}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    scene = _scene(case, seed)
    s = State(case, scene, rzk.AggregateCuda(_context(), scene), seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if "width" in case:
        s.cam = rzk.Camera(scene.camera)
        s.n_recv = s.cam.n_pixels
        s.recv = s.agg.primary(s.cam)
    if "n_vpl" in case:
        s.vpls, emitted = instances.spawn_vpls(s.agg, seed, case["n_vpl"])
        s.scale = 1.0 / emitted
    if "clamp" in case:
        s.ev = rzk.VirtualPointLightCuda(s.agg, MODES[case["clamp"]], TAUS[case["clamp"]])
    if kind == "cluster":
        ev = rzk.VirtualPointLightCuda(s.agg, rzk.CLAMP_RADIANCE, TAUS["radiance"])
        s.a, _ = ev.fill(s.recv, s.n_recv, s.vpls, case["n_vpl"], with_visibility=False)
        s.builder = rzk.ClusterBuilderCuda()
    elif kind == "segments":
        s.a, _ = _surface_points(s, case["n"], gen)
        s.b = _floats(s.vpls)[torch.randint(case["n_vpl"], (case["n"],), generator=gen, device="cuda")][:, 0:3].contiguous()
    elif kind == "rays":
        s.a, n = _surface_points(s, case["n"], gen)
        d = torch.randn(s.a.shape, generator=gen, device="cuda")   # cosine-distributed about the normal
        s.b = (d / d.norm(dim=1, keepdim=True) + 1.0005 * n).contiguous()
    elif kind == "rebuild":
        s.a, _ = _surface_points(s, 20000, gen)
        s.b = s.a.flip(0).contiguous()
    elif kind in ("lightslice", "guided"):
        p = rzk.lightslice_params(num_clusters=case["clusters"], max_slice_size=case["slice"], num_neighbor_slices=32,
                                  max_slice_clusters=case.get("slice_clusters", 1000))
        s.ls = rzk.LightSliceCuda.create(s.agg, s.recv, case["width"], case["height"], s.vpls, case["n_vpl"], p)
    return s


# --------------------------------------------------------------------------------- pass

def _wanted(case):
    """VPLs a frame takes from its particles, the first in push order: fewer than they make."""
    return int(case["particles"] * (1.0 - 0.5 ** (case["bounces"] - 1)))


def run(s):
    if isinstance(s, dict):
        s["batch"].run()
        return [k[3] for k in s["keep"]]
    c = s.case
    kind = c["kind"]
    if kind == "gather":
        return s.ev.gather(s.recv, s.n_recv, s.vpls, c["n_vpl"], scale=s.scale, image_width=c["width"] if c["tiled"] else 0)
    if kind == "fill":
        if c["what"] == "incident":
            return s.ev.incident_radiance(s.recv, s.n_recv, s.vpls, c["n_vpl"])
        return s.ev.fill(s.recv, s.n_recv, s.vpls, c["n_vpl"])
    if kind == "cluster":
        alphas, norms = s.builder.alphas(s.a)
        return [alphas, norms, *s.builder.cluster_by_sampling(s.a, c["clusters"], s.seed)]
    if kind == "segments":
        return s.agg.hit_segments(s.a, s.b)
    if kind == "rays":
        return s.agg.hit_rays(s.a, s.b)
    if kind == "spawn":
        vpls, made = rzk.VplGeneratorCuda(s.agg).spawn(s.seed, c["particles"], c["bounces"])
        return vpls[: _wanted(c) * RECORD], made
    if kind == "lightslice":
        return s.ls.gather(s.recv, s.n_recv, MODES[c["clamp"]], TAUS[c["clamp"]], scale=s.scale)
    if kind == "guided":
        return s.ls.guided_render(s.cam, c["spp"], c["bounces"], rr_depth=3, rr_prob=0.5, seed=s.seed, sampler=c["sampler"])
    s.agg.rebuild()
    return [s.agg.primary(s.cam), s.agg.hit_segments(s.a, s.b)]


# --------------------------------------------------------------------------------- work

def _tris(case):
    return {"room": 36, "objects": 12 + 150 * case["count"], "spheres": 12 + 48 * case["count"]}[case["scene"]]


def _ray(tris):
    """Operations a ray cannot do without: one box test (24) per tree level and one triangle test (40)."""
    return 24 * math.log2(tris + 1) + 40


def work(case):
    kind = case["kind"]
    if kind == "batch":
        pairs = px = 0
        specs = instances.batch_specs(case["jobs"], case["sizes"], tris=(case["tris"] // 3, case["tris"]),
                                      side=(case["side"] // 3, case["side"]), vpls=(case["n_vpl"] // 3, case["n_vpl"]))
        for s in specs:
            pairs += s.width * s.height * s.n_vpl
            px += s.width * s.height
        return {"bytes": px * (RECORD + 12) + sum(s.n_vpl * RECORD + 80 * s.n_tris for s in specs),
                "flops": pairs * (27 + _ray(case["tris"]) / 8)}
    tris = _tris(case)
    scene = 80 * tris   # a triangle record and a tree node each
    n_recv, n_vpl = case.get("width", 0) * case.get("height", 0), case.get("n_vpl", 0)
    pairs = n_recv * n_vpl
    if kind == "gather":      # 27: both facing tests and the form factor; an eighth of the pairs needs a ray
        return {"bytes": scene + n_recv * (RECORD + 12) + n_vpl * RECORD, "flops": pairs * (27 + _ray(tris) / 8)}
    if kind == "fill":
        rays = 0 if case["what"] == "incident" else 1
        return {"bytes": rays * scene + (n_recv + n_vpl) * RECORD + pairs * (12 + rays), "flops": pairs * (27 + rays * _ray(tris))}
    if kind == "cluster":
        return {"bytes": 12 * pairs + 12 * n_vpl, "flops": 6.0 * pairs * case["clusters"] + 12 * pairs}
    if kind == "segments":
        return {"bytes": scene + 25 * case["n"], "flops": case["n"] * _ray(tris)}
    if kind == "rays":
        return {"bytes": scene + case["n"] * (24 + 4 + RECORD), "flops": case["n"] * _ray(tris)}
    if kind == "spawn":
        n = case["particles"]
        return {"bytes": scene + _wanted(case) * RECORD, "flops": n * (case["bounces"] - 1) * (_ray(tris) + 100)}
    if kind == "lightslice":
        return {"bytes": scene + n_recv * (RECORD + 12), "flops": n_recv * case["slice_clusters"] / 2 * (27 + _ray(tris))}
    if kind == "guided":      # at least one light sample, one BRDF sample and one continuation at the first vertex
        return {"bytes": scene + n_recv * 12, "flops": n_recv * case["spp"] * 3 * (_ray(tris) + 100)}
    return {"bytes": 84 * tris + 128 * tris + n_recv * RECORD, "flops": 24 * tris * math.log2(tris) + n_recv * _ray(tris)}


# -------------------------------------------------------------------------------- exact

def _dot(a, b):
    return (a * b).sum(-1)


def _triangles(scene):
    v = torch.from_numpy(scene.prim_v).cuda().double().reshape(-1, 4, 3)
    quad = torch.from_numpy(scene.prim_kind == sg.PRIM_QUAD).cuda()
    return torch.cat([v[:, [0, 1, 2]], v[quad][:, [0, 2, 3]]])


def _tri_t(o, d, tri):
    """Distances [rays, triangles] along unit directions d; inf where a ray misses."""
    e1, e2 = tri[:, 0] - tri[:, 1], tri[:, 0] - tri[:, 2]
    n = torch.linalg.cross(e1, e2)
    denom = d @ n.T                                            # = -(e1 x e2) . -d
    j = tri[None, :, 0] - o[:, None]
    beta = (torch.linalg.cross(j, e2[None].expand_as(j)) * d[:, None]).sum(-1) / denom
    gamma = (torch.linalg.cross(e1[None].expand_as(j), j) * d[:, None]).sum(-1) / denom
    t = (j * n[None]).sum(-1) / denom
    ok = (denom.abs() >= 1e-6) & (beta >= 0) & (gamma >= 0) & (beta + gamma <= 1)
    return torch.where(ok, t, torch.inf)


def _occluded(p, q, tri, tmin):
    out = torch.zeros(p.shape[0], dtype=torch.bool, device="cuda")
    step = max(1, (1 << 22) // tri.shape[0])
    for i in range(0, p.shape[0], step):
        v = q[i:i + step] - p[i:i + step]
        length = v.norm(dim=1, keepdim=True)
        t = _tri_t(p[i:i + step], v / length, tri)
        out[i:i + step] = ((t >= tmin) & (t <= length - tmin)).any(1)
    return out


def _brdf(mats, mat, u, v, n, wo, wi):
    """BRDF values [..., 3] of material indices `mat`."""
    m = mats[mat]
    kind, kd, ks, p0, p1 = m[..., 0], m[..., 1:4], m[..., 4:7], m[..., 7], m[..., 8]
    ci, co = _dot(n, wi), _dot(n, wo)
    lit = (ci > 1e-6) & (co > 1e-6)
    ca = _dot(wo, 2 * ci[..., None] * n - wi)
    phong = torch.where(ca > 0, (p0 + 2) / (2 * math.pi) * ca.clamp_min(1e-300) ** p0, 0.0)
    h = wi + wo
    a, b = torch.where(p0 > 0, p0, 1.0), torch.where(p1 > 0, p1, 1.0)
    expo = torch.exp(-((_dot(u, h) / a) ** 2 + (_dot(v, h) / b) ** 2) / _dot(n, h) ** 2)
    ward = expo / (4 * math.pi * a * b) / (ci * co).clamp_min(1e-300).sqrt()
    spec = torch.where(kind == sg.BSDF_PHONG, phong, torch.where(kind == sg.BSDF_WARD, ward, 0.0))
    return torch.where(lit[..., None], kd / math.pi + ks * spec[..., None], 0.0)


def _materials(scene):
    m = scene.mats
    rows = np.concatenate([m["type"][:, None], m["kd"], m["ks"], m["p0"][:, None], m["p1"][:, None]], 1)
    return torch.from_numpy(rows.astype(np.float64)).cuda()


def _radiance(scene, s, cols, incident):
    """Terms [receivers, cols, 3] without visibility, and the pairs' end points."""
    r, mat = _floats(s.recv).double(), _ints(s.recv)[:, 21].long()
    l, lmat = _floats(s.vpls).double()[cols], _ints(s.vpls)[cols, 21].long()
    mats = _materials(scene)
    p, ns, wo, u, v, n = (r[:, k:k + 3][:, None] for k in ((0, 6, 9, 12, 15, 18) if not incident else (0, 3, 9, 12, 15, 18)))
    q, ln, lu, lv, lnn, lwi, power = (l[:, k:k + 3][None] for k in (0, 3, 6, 9, 12, 15, 18))
    d = q - p
    dd = _dot(d, d)
    g = (_dot(ns, d) * _dot(ln, d)).abs() / dd ** 2
    wi = d / dd.sqrt()[..., None]
    lb = _brdf(mats, lmat.clamp_min(0)[None], lu, lv, lnn, lwi, -wi)
    lb = torch.where((lmat >= 0)[None, :, None], lb, 1.0)
    sb = torch.ones_like(lb) if incident else _brdf(mats, mat.clamp_min(0)[:, None], u, v, n, wo, wi)
    mode, tau = s.case["clamp"], np.float64(np.float32(TAUS[s.case["clamp"]]))
    g = g[..., None]
    if mode == "form_factor":
        x = lb * sb * g.clamp_max(tau) * power
    elif mode == "reflectivity":
        refl = sb * g * lb
        x = refl * (tau / refl.norm(dim=-1, keepdim=True).clamp_min(tau)) * power
    else:
        x = power * g * sb * lb
        if mode == "radiance":
            x = x * (tau / x.norm(dim=-1, keepdim=True).clamp_min(tau))
    if not incident:
        x = torch.where((mat >= 0)[:, None, None], x, 0.0)
    return x, p.expand_as(d), q.expand_as(d)


def _exact_pairs(case, seed):
    """The exact matrix in columns: yields (column range, terms times visibility [receivers, cols, 3])."""
    s = prepare(case, seed)
    tri = _triangles(s.scene)
    incident = case.get("what") == "incident"
    step = max(1, (1 << 20) // s.n_recv)
    for j in range(0, case["n_vpl"], step):
        cols = slice(j, min(case["n_vpl"], j + step))
        x, p, q = _radiance(s.scene, s, cols, incident)
        if not incident:
            lit = (x != 0).any(-1)
            dark = _occluded(p[lit], q[lit], tri, float(np.float32(s.scene.tmin)))
            x[lit] = torch.where(dark[:, None], 0.0, x[lit])
        yield s, cols, x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("gather", "fill"):
        pairs = case["width"] * case["height"] * case["n_vpl"]
        if case.get("what") != "incident" and pairs * _tris(case) > BRUTE:
            return None
        if kind == "gather":
            total = 0.0
            for s, _, x in _exact_pairs(case, seed):
                total = total + x.sum(1)
            return total * np.float64(np.float32(s.scale))
        mat = torch.cat([x.transpose(0, 1) for _, _, x in _exact_pairs(case, seed)])
        return mat if case["what"] == "incident" else (mat, None)
    if kind == "rays" and case["n"] * _tris(case) <= BRUTE:
        s = prepare(case, seed)
        tri, t = _triangles(s.scene), []
        step = max(1, (1 << 22) // tri.shape[0])
        for i in range(0, case["n"], step):
            d = s.b[i:i + step].double()
            x = _tri_t(s.a[i:i + step].double(), d / d.norm(dim=1, keepdim=True), tri)
            x = torch.where(x >= float(np.float32(s.scene.tmin)), x, torch.inf).min(1).values
            t.append(torch.where(x <= 1e6, x, -1.0))
        return torch.cat(t), None
    if kind == "cluster":
        m = prepare(case, seed).a.double()
        mag = m.norm(dim=2)                                    # [cols, rows]
        norm = mag.norm(dim=1)
        return [norm * norm.sum() - mag @ mag.sum(0), norm, None, None, None, None]
    return None
