"""Performance cases of the ray-query engine: what a renderer or a ray server
has the engine do, through the package's public classes.

Kinds of case (`kind`), and what each stands for in use:

  closest  one closest-hit call on device buffers: from a mouse pick or a
           small tile up to the incoherent bounce batch of a whole image.
           `binned` puts the binning pass ahead of the trace.
  any      one any-hit call on device buffers: the shadow rays of a pass.
  host     one call on host buffers (`form` = od: the reference's own Ray
           payload, 24 bytes; rays: 32-byte rays; any: shadow rays), from
           pinned memory: a CPU renderer that hands its rays over.
  kd       the bit-exact parity mode over the kd-tree.
  batch    one launch over many scenes' ray batches, replayed as a graph.
  gather   the radiance estimate of a photon map on device buffers.
  nearest  the k nearest photons of host queries.
  map      a photon map made from photons in device memory, and a gather on
           it: the indirect pass of one frame.
  bounce   eye rays, their hits, hit surfaces, diffuse secondaries and the
           secondaries' hits: one bounce of a path tracer.
  refit    a scene whose triangles moved: the accelerator updated and the
           frame's eye rays traced.

Scenes: `soup` is random triangles in a box 1000 units wide (`tris` of them);
`field` is a square heightfield 1000 units wide (`tris` = 2 * res * res).
The geometry depends on the case alone, like a program's loaded model; rays,
photons, queries and displacements come from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from encore_b200.accel import Accelerator
from encore_b200.batch import BatchLaunch
from encore_b200.photon_map import PhotonMap
from encore_b200.wavefront import camera_rays, diffuse_rays, hit_surface, photon_map_from_device

DEV = "cuda"
SIZE = 1000.0
EYE_SOUP = (0.5 * SIZE, 0.5 * SIZE, -1.5 * SIZE)
EYE_FIELD = (0.503 * SIZE, 1.3 * SIZE, 0.497 * SIZE)


def listed():
    return [
        # a pick or a small tile: launch latency is all there is
        dict(name="closest_tile", kind="closest", scene="soup", tris=10_000, rays=777, mix="eye"),
        # the eye rays of one 1024 x 1024 frame of a small model
        dict(name="closest_frame", kind="closest", scene="soup", tris=10_000, rays=1_048_576,
             mix="eye"),
        # eye rays and diffuse bounces of a large terrain, shuffled
        dict(name="closest_incoherent", kind="closest", scene="field", tris=2_097_152,
             rays=4_179_838, mix="bounce"),
        # the same kind of batch, binned first, on a mid-sized terrain
        dict(name="closest_binned", kind="closest", scene="field", tris=524_288, rays=2_000_001,
             mix="bounce", binned=True),
        # the shadow pass of a frame: about half of the rays blocked
        dict(name="shadow_pass", kind="any", scene="soup", tris=100_000, rays=1_500_007),
        # a CPU renderer's rays, copied in and out
        dict(name="host_rays", kind="host", scene="field", tris=524_288, rays=2_000_003, form="od"),
        # parity with the reference's kd walk
        dict(name="kd_parity", kind="kd", scene="field", tris=524_288, rays=1_000_003, mix="bounce"),
        # a ray server's round over many scenes
        dict(name="batch_scenes", kind="batch", scenes=16, max_tris=100_000, max_rays=500_000),
        # the indirect pass of a photon mapper: k = 50
        dict(name="radiance_50", kind="gather", photons=400_000, queries=300_007, k=50),
        # the frame's photon map made and used
        dict(name="photon_frame", kind="map", photons=500_000, queries=100_003, k=50),
        # one bounce of a path tracer
        dict(name="bounce_frame", kind="bounce", scene="soup", tris=100_000, width=1280, height=720,
             per_hit=2),
        # a moving terrain: update and eye rays
        dict(name="moving_scene", kind="refit", scene="field", tris=524_288, rays=100_003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _field_tris(rng, lo, hi):
    r = _log(rng, lo, hi)
    return 2 * r * r


def draw(rng):
    kind = rng.choice(["closest", "closest", "closest", "any", "host", "kd", "batch", "gather",
                       "nearest", "map", "bounce", "refit"])
    scene = rng.choice(["soup", "field"])
    tris = _log(rng, 500, 200_000) if scene == "soup" else _field_tris(rng, 20, 512)
    c = dict(kind=kind, scene=scene, tris=tris)
    if kind in ("closest", "any", "host", "bounce", "refit"):
        if rng.random() < 0.35:
            c["accel_width"] = rng.choice([2, 4])
        if rng.random() < 0.3:
            c["predicate"] = "noclamp"
    if kind == "closest":
        c.update(rays=_log(rng, 1, 3_000_000), mix=rng.choice(["eye", "bounce"]))
        if rng.random() < 0.3:
            c["binned"] = True
    elif kind == "any":
        c.update(rays=_log(rng, 1, 3_000_000))
    elif kind == "host":
        c.update(rays=_log(rng, 1, 3_000_000), form=rng.choice(["od", "rays", "any"]))
    elif kind == "kd":
        c.update(rays=_log(rng, 100, 1_000_000), mix=rng.choice(["eye", "bounce"]))
        if rng.random() < 0.3:
            c["any"] = True
        elif rng.random() < 0.3:
            c["binned"] = True
    elif kind == "batch":
        c = dict(kind=kind, scenes=rng.randint(2, 20), max_tris=_log(rng, 2_000, 100_000),
                 max_rays=_log(rng, 5_000, 500_000))
    elif kind in ("gather", "nearest", "map"):
        c = dict(kind=kind, photons=_log(rng, 1_000, 500_000),
                 queries=_log(rng, 1, 300_000 if kind != "nearest" else 50_000),
                 k=rng.choice([1, 8, 20, 33, 50, 64, 100, 150, 256]))
        if kind != "nearest" and rng.random() < 0.3:
            c["caustic"] = True
        if rng.random() < 0.3:
            c["ignore_normal"] = True
    elif kind == "bounce":
        c.update(width=_log(rng, 17, 1280), height=_log(rng, 9, 720), per_hit=rng.randint(1, 4))
    elif kind == "refit":
        c.update(rays=_log(rng, 100, 300_000))
        if scene == "field":
            c.pop("accel_width", None)
    return c


# ---------------------------------------------------------------------------
# scenes: float32 arrays in host memory, (tris, 9)

_scenes: dict = {}


def _soup(n, salt=0):
    g = np.random.default_rng(1000 + salt)
    c = g.random((n, 1, 3))
    edge = g.uniform(0.005, 0.05, size=(n, 3, 1))
    u = g.normal(size=(n, 3, 3))
    u /= np.linalg.norm(u, axis=2, keepdims=True)
    return ((c + edge * u) * SIZE).reshape(n, 9).astype(np.float32)


def _field_heights(res):
    """Heights of a (res + 1)^2 grid: six octaves of smoothed value noise."""
    g = torch.Generator().manual_seed(77)
    h = torch.zeros(1, 1, res + 1, res + 1)
    amp, total = 1.0, 0.0
    for o in range(6):
        f = 4 * 2 ** o
        lat = torch.rand(1, 1, f + 2, f + 2, generator=g)
        h += amp * torch.nn.functional.interpolate(lat, (res + 1, res + 1), mode="bicubic",
                                                   align_corners=True)
        total += amp
        amp *= 0.5
    return (0.2 * SIZE / total) * h[0, 0]


def _field_from(y):
    res = y.shape[0] - 1
    t = torch.linspace(0.0, SIZE, res + 1)
    v = torch.stack([t[:, None].expand_as(y), y, t[None, :].expand_as(y)], -1)
    a, b, c, d = v[:-1, :-1], v[1:, :-1], v[1:, 1:], v[:-1, 1:]
    q = torch.stack([torch.cat([a, b, c], -1), torch.cat([a, c, d], -1)], 2)
    return np.ascontiguousarray(q.reshape(-1, 9).float().numpy())


def _scene(case):
    key = (case["scene"], case["tris"])
    if key not in _scenes:
        if len(_scenes) > 6:
            _scenes.clear()
        if case["scene"] == "soup":
            _scenes[key] = _soup(case["tris"])
        else:
            _scenes[key] = _field_from(_field_heights(int(round(math.sqrt(case["tris"] / 2)))))
    return _scenes[key]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _pack(o, d, tmax=math.inf):
    r = torch.empty(o.shape[0], 8, device=o.device)
    r[:, 0:3], r[:, 3], r[:, 4:7], r[:, 7] = o, 0.0, d, tmax
    return r


def _eye_rays(case, n, g):
    """Eye rays through random points of the image, as a jittered camera has them."""
    if case.get("scene") == "field":
        eye, fwd, right, up = EYE_FIELD, (0, -1, 0), (1, 0, 0), (0, 0, 1)
        h = math.tan(math.radians(20.0))
    else:
        eye, fwd, right, up = EYE_SOUP, (0, 0, 1), (1, 0, 0), (0, 1, 0)
        h = math.tan(math.radians(22.5))
    s = (2 * torch.rand(n, 2, device=DEV, generator=g) - 1) * h
    f, r, u = (torch.tensor(v, device=DEV, dtype=torch.float32) for v in (fwd, right, up))
    d = _unit(f + s[:, :1] * r + s[:, 1:] * u)
    return _pack(torch.tensor(eye, device=DEV).expand(n, 3), d)


def _surface(tris, n, g, up_facing):
    """Random points of random triangles and a unit normal on one side."""
    t = torch.from_numpy(tris).to(DEV).view(-1, 3, 3)
    i = torch.randint(0, t.shape[0], (n,), device=DEV, generator=g)
    a, b = torch.rand(2, n, 1, device=DEV, generator=g)
    a = a.sqrt()
    p = (1 - a) * t[i, 0] + a * (1 - b) * t[i, 1] + a * b * t[i, 2]
    nrm = _unit(torch.linalg.cross(t[i, 1] - t[i, 0], t[i, 2] - t[i, 0]))
    if up_facing:
        nrm = torch.where(nrm[:, 1:2] < 0, -nrm, nrm)
    else:
        nrm = torch.where(torch.rand(n, 1, device=DEV, generator=g) < 0.5, -nrm, nrm)
    return p, nrm


def _rays(case, n, g, mix):
    """`eye`: eye rays; `bounce`: a quarter eye rays and three quarters
    cosine-weighted secondaries from surface points, shuffled."""
    ne = n if mix == "eye" else (n + 3) // 4
    rays = _eye_rays(case, ne, g)
    if mix == "eye":
        return rays
    p, nrm = _surface(_scene(case), n - ne, g, case["scene"] == "field")
    d = _unit(nrm + _unit(torch.randn(n - ne, 3, device=DEV, generator=g)) * 0.999)
    rays = torch.cat([rays, _pack(p + 0.1 * nrm, d)])
    return rays[torch.randperm(n, device=DEV, generator=g)].contiguous()


def _shadow_rays(case, n, g):
    p, nrm = _surface(_scene(case), n, g, case["scene"] == "field")
    light = torch.tensor([0.5, 1.4, 0.5], device=DEV) * SIZE
    off = (torch.rand(n, 3, device=DEV, generator=g) - 0.5) * torch.tensor([0.2, 0.0, 0.2], device=DEV)
    v = light + off * SIZE - p
    dist = v.norm(dim=1)
    d = v / dist[:, None]
    return _pack(p + 0.1 * d, d, dist)


def _hits(n):
    """A hit buffer (tri as int32, t u v as float32) and its two halves."""
    h = torch.zeros(n, 4, dtype=torch.int32, device=DEV)
    return h, {"tri": h[:, 0], "tuv": h.view(torch.float32)[:, 1:]}


# Photons of a closed room: its six walls and three shelves, axis-aligned like
# the boxes photon maps are drawn with; denser under the light.  A query
# lies on a wall and carries that wall's normal.
def _room_points(n, g):
    wall = torch.randint(0, 9, (n,), device=DEV, generator=g)
    uv = torch.rand(n, 2, device=DEV, generator=g)
    uv = torch.where(torch.rand(n, 1, device=DEV, generator=g) < 0.3, 0.35 + 0.3 * uv, uv) * SIZE
    axis = wall % 3
    level = torch.tensor([0.0, 1.0, 0.4], device=DEV)[wall // 3] * SIZE
    p = torch.empty(n, 3, device=DEV)
    for a in range(3):
        m = axis == a
        p[m, a] = level[m]
        p[m, (a + 1) % 3] = uv[m, 0]
        p[m, (a + 2) % 3] = uv[m, 1]
    nrm = torch.nn.functional.one_hot(axis, 3).float()
    nrm = torch.where((wall // 3 == 1)[:, None], -nrm, nrm) + 0.0
    return p, nrm


def _photons(case, seed):
    """Photon positions, normals and powers, query points and normals, and the
    search radius: wide enough that a query in an even map finds about 1.2 k
    photons, and at most a fifth of the room."""
    g = _gen(seed)
    n, q = case["photons"], case["queries"]
    pos, nrm = _room_points(n, g)
    power = torch.rand(n, 3, device=DEV, generator=g) / n
    qpos, qnrm = _room_points(q, g)
    r = min(0.2 * SIZE, SIZE * math.sqrt(1.2 * case["k"] * 9 / (math.pi * n)))
    return pos, nrm, power, qpos, qnrm, float(np.float32(r))


def _accel(case, kind="wbvh"):
    return Accelerator(kind, width=case.get("accel_width", 8),
                       predicate=case.get("predicate", "reference")).build(_scene(case))


def _batch_sizes(case):
    n = case["scenes"]
    rays = np.exp(np.random.default_rng(9).uniform(math.log(4_096), math.log(max(4_097, case["max_rays"])), n)).astype(int)
    t = np.random.default_rng(5)
    tris = np.exp(t.uniform(math.log(1_000), math.log(max(1_001, case["max_tris"])), n)).astype(int)
    rays[0], tris[0] = case["max_rays"], case["max_tris"]
    return tris, rays


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    s = {"kind": kind, "case": case}
    if kind in ("closest", "kd", "any"):
        n = case["rays"]
        s["acc"] = _accel(case, "kdtree" if kind == "kd" else "wbvh")
        if kind == "any" or case.get("any"):
            s["rays"] = _shadow_rays(case, n, g)
            s["occ"] = torch.zeros(n, dtype=torch.uint8, device=DEV)
            s["kind"] = "any"
        else:
            s["rays"] = _rays(case, n, g, case["mix"])
            s["hits"], s["out"] = _hits(n)
            s["kind"] = "closest"
        if case.get("binned"):
            s["scratch"] = torch.empty(s["acc"].bin_scratch_bytes(n), dtype=torch.uint8, device=DEV)
    elif kind == "host":
        n, form = case["rays"], case["form"]
        s["acc"] = _accel(case)
        rays = _shadow_rays(case, n, g) if form == "any" else _rays(case, n, g, "bounce")
        if form == "od":
            rays = torch.cat([rays[:, 0:3], rays[:, 4:7]], 1)
        s["rays"] = torch.empty(rays.shape, pin_memory=True).copy_(rays)
        if form == "any":
            s["res"] = torch.zeros(n, dtype=torch.uint8, pin_memory=True)
            s["out"] = s["res"]
        else:
            s["res"] = torch.zeros(n, 4, dtype=torch.int32, pin_memory=True)
            s["out"] = {"tri": s["res"][:, 0], "tuv": s["res"].view(torch.float32)[:, 1:]}
    elif kind == "batch":
        items, outs = [], []
        for i, (nt, nr) in enumerate(zip(*_batch_sizes(case))):
            c = dict(scene="soup", tris=int(nt))
            acc = Accelerator("wbvh").build(_soup(int(nt), salt=i))
            rays = torch.cat([_eye_rays(c, int(nr) // 2, g), _inside_rays(int(nr) - int(nr) // 2, g)])
            rays = rays[torch.randperm(int(nr), device=DEV, generator=g)].contiguous()
            h, out = _hits(int(nr))
            items.append((acc, rays, h))
            outs.append(out)
        s["batch"], s["out"] = BatchLaunch(items), outs
    elif kind in ("gather", "map", "nearest"):
        pos, nrm, power, qpos, qnrm, s["r"] = _photons(case, seed)
        if kind == "map":
            s["photons"] = (pos, nrm, power)
        else:
            s["map"] = PhotonMap(len(pos), caustic=case.get("caustic", False))
            s["map"].add_photons(pos.cpu().numpy(), nrm.cpu().numpy(), power.cpu().numpy())
            s["map"].balance_and_construct()
        if kind == "nearest":
            s["q"], s["qn"] = qpos.cpu().numpy(), qnrm.cpu().numpy()
        else:
            s["q"], s["qn"] = qpos, qnrm
            s["rgb"] = torch.zeros_like(qpos)
    elif kind == "bounce":
        n = case["width"] * case["height"]
        m = n * case["per_hit"]
        s["acc"] = _accel(case)
        s["rays"] = torch.zeros(n, 8, device=DEV)
        s["hits"], out1 = _hits(n)
        s["pos"], s["nrm"] = torch.zeros(n, 3, device=DEV), torch.zeros(n, 3, device=DEV)
        s["sec"] = torch.zeros(m, 8, device=DEV)
        s["hits2"], out2 = _hits(m)
        s["seed"] = int(seed) % 100_000 + 1
        s["out"] = {"rays": s["rays"], "hits": out1, "pos": s["pos"], "nrm": s["nrm"],
                    "sec": s["sec"], "hits2": out2}
    elif kind == "refit":
        s["acc"] = _accel(case)
        s["moved"] = _moved(case, seed)
        s["rays"] = _eye_rays(case, case["rays"], g)
        s["hits"], s["out"] = _hits(case["rays"])
    return s


def _inside_rays(n, g):
    o = torch.rand(n, 3, device=DEV, generator=g) * SIZE
    return _pack(o, _unit(torch.randn(n, 3, device=DEV, generator=g)))


def _moved(case, seed):
    """The scene's triangles a little later: a wave through the field, or every
    triangle of the soup drifted by a few units."""
    t = _scene(case)
    r = np.random.default_rng(seed)
    if case["scene"] == "soup":
        return t + np.tile(r.uniform(-8.0, 8.0, (len(t), 3)).astype(np.float32), (1, 3))
    v = t.reshape(-1, 3, 3).copy()
    k, ph = r.uniform(0.005, 0.03, 2), r.uniform(0, 6.28, 2)
    v[..., 1] += (12.0 * np.sin(k[0] * v[..., 0] + ph[0]) * np.cos(k[1] * v[..., 2] + ph[1])
                  ).astype(np.float32)
    return v.reshape(-1, 9)


def run(s):
    kind = s["kind"]
    if kind == "closest":
        n = s["rays"].shape[0]
        if "scratch" in s:
            s["acc"].intersect_device_binned(s["rays"], n, s["hits"], s["scratch"])
        else:
            s["acc"].intersect_device(s["rays"], n, s["hits"])
        return s["out"]
    if kind == "any":
        s["acc"].occluded_device(s["rays"], s["rays"].shape[0], s["occ"])
        return s["occ"]
    if kind == "host":
        form = s["case"]["form"]
        if form == "od":
            s["acc"].intersect_od(s["rays"], out=s["res"])
        elif form == "rays":
            s["acc"].intersect(s["rays"], out=s["res"])
        else:
            s["acc"].occluded(s["rays"], out=s["res"])
        return s["out"]
    if kind == "batch":
        s["batch"].launch_graph()
        return s["out"]
    c = s["case"]
    ign = c.get("ignore_normal", False)
    if kind == "gather":
        s["map"].get_radiance_estimate_device(c["k"], s["r"], s["q"], s["qn"], s["q"].shape[0],
                                              s["rgb"], ignore_normal=ign)
        return s["rgb"]
    if kind == "nearest":
        idx, d2, cnt = s["map"].get_nearest_n_photons(c["k"], s["r"], s["q"], s["qn"],
                                                      ignore_normal=ign)
        return {"idx": idx, "d2": d2, "count": cnt}
    if kind == "map":
        pos, nrm, power = s["photons"]
        pm = photon_map_from_device(pos, nrm, power, pos.shape[0], caustic=c.get("caustic", False))
        pm.get_radiance_estimate_device(c["k"], s["r"], s["q"], s["qn"], s["q"].shape[0], s["rgb"],
                                        ignore_normal=ign)
        return s["rgb"]
    if kind == "bounce":
        acc, n = s["acc"], s["rays"].shape[0]
        eye, look, up, fov = _camera(c)
        camera_rays(eye, look, up, fov, c["width"], c["height"], s["rays"], jitter_seed=s["seed"])
        acc.intersect_device(s["rays"], n, s["hits"])
        hit_surface(acc, s["hits"], n, s["pos"], s["nrm"])
        diffuse_rays(acc, s["rays"], s["hits"], n, c["per_hit"], s["seed"], 0.1, s["sec"])
        acc.intersect_device(s["sec"], n * c["per_hit"], s["hits2"])
        return s["out"]
    if kind == "refit":
        s["acc"].update(s["moved"])
        s["acc"].intersect_device(s["rays"], s["rays"].shape[0], s["hits"])
        return s["out"]
    raise ValueError(kind)


def _camera(case):
    if case["scene"] == "field":
        return EYE_FIELD, (0.503 * SIZE, 0.0, 0.497 * SIZE), (0.0, 0.0, 1.0), 40.0
    return EYE_SOUP, (0.5 * SIZE, 0.5 * SIZE, 0.5 * SIZE), (0.0, 1.0, 0.0), 45.0


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _trace_work(n, ntris, ray=32, hit=16):
    """Each ray read and each result written once; of the scene what n rays can
    touch at most (a triangle's 36 bytes each).  Per ray one path of eight-wide
    box tests from root to leaf and two triangle tests."""
    levels = math.log(max(ntris, 2), 8)
    return n * (ray + hit) + 36 * min(ntris, 2 * n), n * (levels * 8 * 12 + 2 * 50)


def work(case):
    kind = case["kind"]
    if kind in ("closest", "kd", "any", "host"):
        is_any = kind == "any" or case.get("any") or case.get("form") == "any"
        b, f = _trace_work(case["rays"], case["tris"], 24 if case.get("form") == "od" else 32,
                           1 if is_any else 16)
    elif kind == "batch":
        b = f = 0
        for nt, nr in zip(*_batch_sizes(case)):
            x, y = _trace_work(int(nr), int(nt))
            b, f = b + x, f + y
    elif kind in ("gather", "nearest", "map"):
        q, n, k = case["queries"], case["photons"], case["k"]
        out = 12 if kind != "nearest" else 4 + 8 * k
        b = q * (24 + out) + (36 * n if kind == "map" else 36 * min(n, q * k))
        f = q * 2 * k * 9
        if kind == "map":
            f += n * math.log2(max(2, n / 32)) * 4
    elif kind == "bounce":
        n = case["width"] * case["height"]
        m = n * case["per_hit"]
        b1, f1 = _trace_work(n, case["tris"])
        b2, f2 = _trace_work(m, case["tris"])
        b, f = b1 + b2 + 24 * n, f1 + f2 + n * 60 + m * 120
    else:
        b, f = _trace_work(case["rays"], case["tris"])
        b, f = b + 36 * case["tris"], f + 40 * case["tris"]
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------
# the same in 64 bits

MOST_PAIRS = 6.0e10


def _closest64(tris, rays):
    """Closest hit of every ray by testing every triangle (t, u, v; 0 for a
    miss): the numerators and the determinant of the Moller-Trumbore test as
    products of per-ray and per-triangle vectors."""
    t = torch.from_numpy(tris).to(DEV).double().view(-1, 3, 3)
    v0, e1, e2 = t[:, 0], t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    ka = torch.cat([e2, -torch.linalg.cross(e2, v0)], 1).T.contiguous()
    kb = torch.cat([-e1, -torch.linalg.cross(v0, e1)], 1).T.contiguous()
    kd = (-nrm).T.contiguous()
    kt = torch.cat([nrm, -(v0 * nrm).sum(1, keepdim=True)], 1).T.contiguous()
    out = torch.zeros(rays.shape[0], 3, dtype=torch.float64, device=DEV)
    step = max(1, int(2.5e8 // t.shape[0]))
    for b in range(0, rays.shape[0], step):
        r = rays[b:b + step].double()
        o, d = r[:, 0:3], r[:, 4:7]
        md = torch.cat([torch.linalg.cross(o, d), d], 1)
        inv = 1.0 / (d @ kd)
        al, be = (md @ ka) * inv, (md @ kb) * inv
        tt = (torch.cat([o, torch.ones_like(o[:, :1])], 1) @ kt) * inv
        bad = ~((al >= 0) & (be >= 0) & (al + be <= 1) & (tt > r[:, 3:4]) & (tt < r[:, 7:8]))
        tt = tt.masked_fill_(bad, math.inf)
        best, i = tt.min(1, keepdim=True)
        hit = torch.isfinite(best)
        res = torch.cat([best, al.gather(1, i), be.gather(1, i)], 1)
        out[b:b + step] = torch.where(hit, res, torch.zeros_like(res))
    return out


def _radiance64(case, seed):
    pos, nrm, power, qpos, qnrm, r = _photons(case, seed)
    k = min(case["k"], pos.shape[0])
    p, pw = pos.double(), power.double()
    out = torch.zeros(qpos.shape[0], 3, dtype=torch.float64, device=DEV)
    caustic = case.get("caustic", False)
    step = max(1, int(2.5e8 // pos.shape[0]))
    for b in range(0, qpos.shape[0], step):
        q = qpos[b:b + step].double()
        d2 = torch.zeros(q.shape[0], p.shape[0], dtype=torch.float64, device=DEV)
        for a in range(3):
            d2 += (q[:, a:a + 1] - p[None, :, a]).square_()
        off = d2 >= r * r
        if not case.get("ignore_normal", False):
            for a in range(3):
                off |= qnrm[b:b + step, a:a + 1] != nrm[None, :, a]
        d2.masked_fill_(off, math.inf)
        near, i = d2.topk(k, dim=1, largest=False)
        has = torch.isfinite(near)
        far = torch.where(has, near, torch.zeros_like(near)).max(1, keepdim=True).values
        w = torch.where(has, (far - near) / near if caustic else torch.ones_like(near),
                        torch.zeros_like(near))
        rgb = (pw[i] * w[..., None]).sum(1)
        if caustic:
            rgb = torch.where(has.any(1, keepdim=True), rgb * (case["k"] / (3.14159 * far * far)), rgb)
        out[b:b + step] = rgb
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "closest" and case["rays"] * case["tris"] <= MOST_PAIRS:
        rays = _rays(case, case["rays"], _gen(seed), case["mix"])
        return {"tri": None, "tuv": _closest64(_scene(case), rays)}
    if kind == "host" and case["form"] != "any" and case["rays"] * case["tris"] <= MOST_PAIRS:
        rays = _rays(case, case["rays"], _gen(seed), "bounce")
        return {"tri": None, "tuv": _closest64(_scene(case), rays)}
    if kind == "refit" and case["rays"] * case["tris"] <= MOST_PAIRS:
        rays = _eye_rays(case, case["rays"], _gen(seed))
        return {"tri": None, "tuv": _closest64(_moved(case, seed), rays)}
    if kind in ("gather", "map") and case["queries"] * case["photons"] <= 3 * MOST_PAIRS:
        return _radiance64(case, seed)
    return None
