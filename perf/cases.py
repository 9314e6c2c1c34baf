"""Performance cases of the ray-query library: what a program that uses it has it do.

Every case goes through the public entry points of `crt_gb300.lib` (contexts, scenes, queries, batches).
A case names its kind, its scene and its sizes:

  closest / any   explicit rays on device buffers (crt_trace_closest / crt_trace_any)
  passes          depth, instance and normal passes of one camera into numpy arrays (crt_passes)
  lidar           one beam-grid scan into device buffers (crt_lidar_grid)
  render          one render into device buffers (crt_render)
  mixed           renders, scans and radiation-pressure queries in one call (crt_batch_mixed)
  srp             force, torque and facet power over a sun-ray grid (crt_srp)
  rebuild         scene build from triangles in host memory, one camera's passes, scene release: what a
                  program with moving bodies does for every frame

The bodies are the repository's own: the procedural asteroid, the spacecraft and the Cornell box.  The
seed gives the body's pose and everything about the request: rays, camera, sun, beams, attitudes.
"""
import functools
import itertools
import math
import os
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (REPO, os.path.join(REPO, "ceres-raytracer_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from crt_gb300 import lib, scenes  # noqa: E402

SUN_DISTANCE = 1.0e9
FLT_MAX = 3.402823466e38


def listed():
    return [
        # a handful of line-of-sight checks in a planning loop: latency
        dict(name="closest_rays_256", kind="closest", body="asteroid", faces=20_000, n=256),
        # incoherent rays on the benchmark's body: secondary rays of a user's own integrator
        dict(name="closest_rays_3m", kind="closest", body="asteroid", faces=2_000_000, n=3_000_017),
        # sun visibility of a set of surface points
        dict(name="any_rays_333k", kind="any", body="asteroid", faces=100_000, n=333_333),
        # depth / id / normal images of a smooth-shaded body for a navigation filter, host results
        dict(name="passes_1021x767", kind="passes", body="asteroid", faces=20_000, smooth=True, width=1021, height=767),
        # the benchmark's LiDAR scan
        dict(name="lidar_1024", kind="lidar", body="asteroid", faces=2_000_000, nx=1024, ny=1024),
        # a thumbnail render in a loop: launches count
        dict(name="render_128", kind="render", body="asteroid", faces=100_000, width=128, height=128, spp=1, bounces=1),
        # the benchmark's render: primary and sun-shadow rays
        dict(name="render_2048", kind="render", body="asteroid", faces=2_000_000, width=2048, height=2048, spp=1,
             bounces=1),
        # the Cornell box path trace of the benchmark
        dict(name="render_cornell_256", kind="render", body="cornell", faces=36, width=256, height=256, spp=16,
             bounces=3),
        # many clients' requests as one call: multi-bounce renders, scans, radiation pressure
        dict(name="mixed_batch_24", kind="mixed", body="asteroid", faces=500_000, n_render=12, n_lidar=8, n_srp=4,
             res=512, spp=4, bounces=2),
        # one attitude of a propagation step
        dict(name="srp_1x250", kind="srp", body="spacecraft", faces=48_728, n_att=1, grid=250, bounces=2),
        # an attitude table of a spacecraft with facet powers
        dict(name="srp_12x2048", kind="srp", body="spacecraft", faces=48_728, n_att=12, grid=2048, bounces=2,
             facets=True),
        # a moving body: build, one camera's passes, release
        dict(name="rebuild_500k", kind="rebuild", body="asteroid", faces=500_000, sah=True, width=640, height=480),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest", "any", "passes", "lidar", "render", "cornell", "mixed", "srp", "rebuild"])
    faces = 2 * _log_int(rng, 1_000, 500_000)   # a closed triangle mesh has an even number of faces
    if kind in ("closest", "any"):
        return dict(kind=kind, body="asteroid", faces=faces, n=_log_int(rng, 100, 3_000_000))
    if kind == "passes":
        return dict(kind=kind, body="asteroid", faces=2 * _log_int(rng, 1_000, 50_000), smooth=rng.random() < 0.5,
                    width=_log_int(rng, 32, 1500), height=_log_int(rng, 32, 1500))
    if kind == "lidar":
        return dict(kind=kind, body="asteroid", faces=faces, nx=_log_int(rng, 16, 1024), ny=_log_int(rng, 16, 1024))
    if kind == "render":
        spp = rng.choice([1, 2, 4])
        return dict(kind=kind, body="asteroid", faces=faces, width=_log_int(rng, 32, 1024),
                    height=_log_int(rng, 32, 1024), spp=spp, bounces=rng.choice([1, 2]))
    if kind == "cornell":
        return dict(kind="render", body="cornell", faces=36, width=_log_int(rng, 32, 512),
                    height=_log_int(rng, 32, 512), spp=rng.choice([1, 4, 16]), bounces=rng.choice([1, 2, 3]))
    if kind == "mixed":
        return dict(kind=kind, body="asteroid", faces=faces, n_render=rng.randint(1, 12), n_lidar=rng.randint(1, 8),
                    n_srp=rng.randint(1, 4), res=_log_int(rng, 64, 512), spp=rng.choice([1, 2, 4]), bounces=2)
    if kind == "srp":
        return dict(kind=kind, body="spacecraft", faces=48_728, n_att=rng.randint(1, 8), grid=_log_int(rng, 64, 2048),
                    bounces=rng.choice([0, 1, 2]), facets=rng.random() < 0.5)
    return dict(kind=kind, body="asteroid", faces=2 * _log_int(rng, 1_000, 250_000), sah=rng.random() < 0.5,
                width=_log_int(rng, 64, 640), height=_log_int(rng, 64, 480))


# ---------------------------------------------------------------- scenes
class _Soup:
    """A mesh already laid out as triangles, as a program keeps it between builds."""

    def __init__(self, mesh, smooth=False):
        self.xyz = mesh.soup()
        self.n_tris = mesh.n_tris
        self.vn = mesh.soup_normals().astype(np.float32) if smooth else None

    def soup(self):
        return self.xyz

    def soup_normals(self):
        return self.vn


@functools.lru_cache(maxsize=None)
def _asteroid(faces, smooth):
    return _Soup(scenes.asteroid(faces, seed=0), smooth)


@functools.lru_cache(maxsize=None)
def _spacecraft():
    return [(e.name, _Soup(e.mesh), e.color, e.rho_s, e.rho_d) for e in scenes.spacecraft()]


@functools.lru_cache(maxsize=None)
def _context(sah=True):
    """The process's context (one more with the fast-build setting of the per-frame path)."""
    ctx = lib.Context(0)
    if not sah:
        ctx.set_tuning(build_sah=False, treelet_passes=0)
    return ctx


def _entities(case, rng):
    """Entity list of a case; the body turned by a random rotation."""
    R = scenes.quaternion_to_matrix(scenes.random_quaternions(1, int(rng.integers(1 << 30)))[0])
    if case["body"] == "asteroid":
        m = _asteroid(case["faces"], bool(case.get("smooth", False)))
        return [scenes.EntitySpec("asteroid", m, (0.1, 0.1, 0.1), smooth=bool(case.get("smooth", False)), rotation=R,
                                  rho_s=0.0, rho_d=0.1)]
    if case["body"] == "spacecraft":
        return [scenes.EntitySpec(n, m, c, rotation=R, rho_s=s, rho_d=d) for n, m, c, s, d in _spacecraft()]
    return scenes.cornell()[0]


def _unit(rng):
    v = rng.normal(size=3)
    return v / np.linalg.norm(v)


def _camera(rng, w, h, rmin=3000.0, rmax=10000.0, frame=1100.0):
    """Camera on a shell around the asteroid that frames the body; square pixels."""
    pos = _unit(rng) * rng.uniform(rmin, rmax)
    cam = scenes.fov_camera(frame / np.linalg.norm(pos), (w, h), pos, (0.0, 0.0, 0.0))
    s = cam["sensor_size"][0]
    cam["sensor_size"] = [s * w / max(w, h), s * h / max(w, h)]
    return cam


def _sun(rng):
    return [dict(type="point", intensity=SUN_DISTANCE ** 2, position=SUN_DISTANCE * _unit(rng))]


def _rays(case, rng):
    """[n, 8] float32 rays (origin, tmin, direction, tmax): from points around the body towards points
    on it or just past its limb (closest), from points near its surface towards a sun (any)."""
    n = case["n"]
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    r = np.empty((n, 8), np.float32)
    if case["kind"] == "closest":
        o = u * rng.uniform(1500.0, 6000.0, (n, 1))
        t = rng.normal(size=(n, 3))
        t *= (1100.0 * rng.uniform(0.0, 1.0, (n, 1)) ** (1 / 3)) / np.linalg.norm(t, axis=1)[:, None]
        d = t - o
        d /= np.linalg.norm(d, axis=1)[:, None]
    else:
        o = u * rng.uniform(1000.0, 1100.0, (n, 1))
        d = np.broadcast_to(_unit(rng), (n, 3))
    r[:, 0:3], r[:, 3], r[:, 4:7], r[:, 7] = o, 0.0, d, FLT_MAX
    return r


def _srp_request(case, rng, n_att):
    return dict(sun_dir=_unit(rng), quaternions=scenes.random_quaternions(n_att, int(rng.integers(1 << 30))),
                grid=int(case["grid"]), num_bounces=int(case["bounces"]), center_of_mass=(0.1, -0.05, 0.02))


def _mixed_requests(case, rng):
    """Sizes by the request's place in the list (the resolution, a half or a quarter of it); the kinds
    take turns."""
    renders, scans, srps = [], [], []
    for i in range(case["n_render"]):
        res = max(16, case["res"] >> (i % 3))
        renders.append(dict(kind="render", camera=_camera(rng, res, res), lights=_sun(rng), min_samples=case["spp"],
                            max_samples=case["spp"], noise_threshold=0.0, num_bounces=case["bounces"],
                            seed=int(rng.integers(1 << 30)), request=i, radiance=True))
    for i in range(case["n_lidar"]):
        m = max(16, case["res"] >> (i % 3))
        pos = _unit(rng) * rng.uniform(3000.0, 10000.0)
        scans.append(dict(kind="lidar", position=pos, rotation=scenes.look_at(pos, (0.0, 0.0, 0.0)), nx=m, ny=m,
                          half_x=math.radians(5.0), half_y=math.radians(5.0)))
    for i in range(case["n_srp"]):
        q = _srp_request(dict(grid=max(16, case["res"] >> (i % 2)), bounces=2), rng, 1)
        srps.append(dict(q, kind="srp", center_of_mass=(0.0, 0.0, 0.0)))
    turns = itertools.zip_longest(renders, scans, srps)
    return [r for t in turns for r in t if r is not None]


def _request(case, seed):
    """Everything about a case that comes from the seed, on the host."""
    rng = np.random.Generator(np.random.PCG64(seed))
    q = dict(entities=_entities(case, rng))
    kind = case["kind"]
    if kind in ("closest", "any"):
        q["rays"] = _rays(case, rng)
    elif kind in ("passes", "rebuild"):
        q["camera"] = _camera(rng, case["width"], case["height"])
    elif kind == "lidar":
        pos = 5000.0 * _unit(rng)
        q["scan"] = dict(position=pos, rotation=scenes.look_at(pos, (0.0, 0.0, 0.0)), nx=case["nx"], ny=case["ny"],
                         half_x=math.radians(5.0), half_y=math.radians(5.0))
    elif kind == "render":
        q["seed"] = int(rng.integers(1 << 30))
        if case["body"] == "cornell":
            _, cam, lights = scenes.cornell()
            cam = dict(cam, resolution=[case["width"], case["height"]],
                       position=cam["position"] + 0.05 * rng.normal(size=3))
            q["camera"], q["lights"] = cam, lights
        else:
            q["camera"], q["lights"] = _camera(rng, case["width"], case["height"]), _sun(rng)
    elif kind == "srp":
        q["srp"] = _srp_request(case, rng, case["n_att"])
    elif kind == "mixed":
        q["requests"] = _mixed_requests(case, rng)
    return q


def prepare(case, seed):
    q = _request(case, seed)
    kind = case["kind"]
    st = dict(case=case, q=q)
    dev = dict(device="cuda")
    if kind == "rebuild":
        st["ctx"] = _context(bool(case["sah"]))
        return st
    ctx = st["ctx"] = _context()
    scene = st["scene"] = ctx.scene(q["entities"])
    if kind in ("closest", "any"):
        n = case["n"]
        st["rays"] = torch.from_numpy(q["rays"]).cuda()
        st["out"] = torch.empty((n, 4), dtype=torch.float32, **dev) if kind == "closest" else \
            torch.empty(n, dtype=torch.uint8, **dev)
    elif kind == "lidar":
        shape = (case["ny"], case["nx"])
        st["range"] = torch.empty(shape, dtype=torch.float64, **dev)
        st["prim"] = torch.empty(shape, dtype=torch.int32, **dev)
    elif kind == "render":
        shape = (case["height"], case["width"], 4)
        st["rgba"] = torch.empty(shape, dtype=torch.uint8, **dev)
        st["radiance"] = torch.empty(shape, dtype=torch.float32, **dev)
    elif kind == "srp":
        n = case["n_att"]
        st["quaternions"] = np.ascontiguousarray(q["srp"]["quaternions"])
        st["force"] = torch.empty((n, 3), dtype=torch.float64, **dev)
        st["torque"] = torch.empty((n, 3), dtype=torch.float64, **dev)
        st["facets"] = torch.empty((n, scene.stats()["n_tris"]), dtype=torch.float64, **dev) \
            if case.get("facets") else None
    elif kind == "mixed":
        outs = []
        for r in q["requests"]:
            r["scene"] = scene
            if r["kind"] == "render":
                w, h = r["camera"]["resolution"]
                outs.append((torch.empty((h, w, 4), dtype=torch.uint8, **dev),
                             torch.empty((h, w, 4), dtype=torch.float32, **dev)))
            elif r["kind"] == "lidar":
                outs.append((torch.empty((r["ny"], r["nx"]), dtype=torch.float64, **dev),
                             torch.empty((r["ny"], r["nx"]), dtype=torch.int32, **dev)))
            else:
                outs.append((torch.empty((1, 3), dtype=torch.float64, **dev),
                             torch.empty((1, 3), dtype=torch.float64, **dev)))
        st["outs"] = outs
    return st


def run(st):
    case, q = st["case"], st["q"]
    kind = case["kind"]
    if kind == "closest":
        out = st["scene"].trace_closest(st["rays"], st["out"])
        return out[:, :3], out.view(torch.int32)[:, 3]
    if kind == "any":
        return st["scene"].trace_any(st["rays"], st["out"])
    if kind == "passes":
        return st["scene"].passes(q["camera"])
    if kind == "lidar":
        s = q["scan"]
        return st["scene"].lidar_grid(s["position"], s["rotation"], s["nx"], s["ny"], s["half_x"], s["half_y"],
                                      out_range=st["range"], out_prim=st["prim"])
    if kind == "render":
        return st["scene"].render(q["camera"], q["lights"], case["spp"], case["spp"], 0.0, case["bounces"],
                                  seed=q["seed"], out_rgba=st["rgba"], out_radiance=st["radiance"])
    if kind == "srp":
        s = q["srp"]
        st["scene"].srp_into(s["sun_dir"], st["quaternions"], s["grid"], st["force"], st["torque"], st["facets"],
                             num_bounces=s["num_bounces"], center_of_mass=s["center_of_mass"])
        return [st["force"], st["torque"], st["facets"]]
    if kind == "mixed":
        outs, _ = st["ctx"].batch(q["requests"], outputs=st["outs"])
        return [list(o) for o in outs]
    scene = st["ctx"].scene(q["entities"])
    out = scene.passes(q["camera"])
    scene.close()
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: the scene's triangles (three FP32 vertices), the rays where they are given, and the outputs.
    Operations: per ray the boxes of one path down a balanced 8-wide tree (8 x 15 operations a level) and
    one triangle test (~45); every camera path's bounces and shadow rays count as rays."""
    kind, faces = case["kind"], case["faces"]
    per_ray = math.ceil(math.log(max(faces, 8), 8)) * 8 * 15 + 45
    tri = 36 * faces
    if kind == "closest":
        rays, data = case["n"], 48 * case["n"]
    elif kind == "any":
        rays, data = case["n"], 33 * case["n"]
    elif kind in ("passes", "rebuild"):
        rays = case["width"] * case["height"]
        data = 52 * rays
    elif kind == "lidar":
        rays = case["nx"] * case["ny"]
        data = 12 * rays
    elif kind == "render":
        pix = case["width"] * case["height"]
        rays = pix * case["spp"] * 2 * case["bounces"]
        data = 20 * pix
    elif kind == "srp":
        rays = case["n_att"] * case["grid"] ** 2
        data = case["n_att"] * (80 + (8 * faces if case.get("facets") else 0))
    else:   # renders and scans at a mean size (the resolution or a half or a quarter of it)
        pix = case["res"] ** 2 * (1 + 1 / 4 + 1 / 16) / 3
        rays = case["n_render"] * pix * case["spp"] * 2 * case["bounces"] + case["n_lidar"] * pix + \
            case["n_srp"] * case["res"] ** 2 * (1 + 1 / 4) / 2
        data = case["n_render"] * pix * 20 + case["n_lidar"] * pix * 12
    return dict(bytes=tri + data, flops=rays * per_ray)


# ---------------------------------------------------------------- the same in 64 bits
def _triangles(entities):
    """FP64 triangles (p0, p1, p2), per-corner normals where shaded smoothly, and the entity of each."""
    P, N, E = [], [], []
    for i, e in enumerate(entities):
        R = torch.as_tensor(np.asarray(e.rotation, np.float64)).cuda()
        t = torch.as_tensor(np.asarray(e.position, np.float64)).cuda()
        p = torch.as_tensor(np.asarray(e.mesh.soup())).cuda().double().reshape(-1, 3, 3)
        P.append((p * e.scale) @ R.T + t)
        vn = torch.as_tensor(np.asarray(e.mesh.soup_normals())).cuda().double().reshape(-1, 3, 3) @ R.T \
            if e.smooth else torch.zeros_like(p)
        N.append(vn)
        E.append(torch.full((p.shape[0],), i, dtype=torch.long, device="cuda"))
    return torch.cat(P), torch.cat(N), torch.cat(E)


def _first_hit(P, o, d, skip=None, pairs=1 << 25):
    """Closest hit of rays (o, d) on triangles P by testing every pair, in Pluecker form: per ray the
    distance (inf: none), the triangle, and the barycentrics (u of p1, v of p2)."""
    e1, e2 = P[:, 0] - P[:, 1], P[:, 2] - P[:, 0]
    n = torch.linalg.cross(e1, e2)
    B2 = torch.cat([torch.linalg.cross(P[:, 0], e2), -e2], 1).T   # (d x (p0 - o)) . e2
    B1 = torch.cat([torch.linalg.cross(P[:, 0], e1), -e1], 1).T
    np0 = (n * P[:, 0]).sum(1)
    R, T = o.shape[0], P.shape[0]
    t_out = torch.full((R,), math.inf, dtype=torch.float64, device=o.device)
    k_out = torch.zeros(R, dtype=torch.long, device=o.device)
    step = max(1, pairs // max(T, 1))
    for a in range(0, R, step):
        oo, dd = o[a:a + step], d[a:a + step]
        L = torch.cat([dd, torch.linalg.cross(dd, oo)], 1)
        den = dd @ n.T
        u = (L @ B2) / den
        v = (L @ B1) / den
        t = (np0[None] - oo @ n.T) / den
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0)
        if skip is not None:
            ok[torch.arange(oo.shape[0], device=o.device), skip[a:a + step]] = False
        t = torch.where(ok, t, math.inf)
        t_out[a:a + step], k_out[a:a + step] = t.min(1)
    k = k_out
    L = torch.cat([d, torch.linalg.cross(d, o)], 1)
    den = (d * n[k]).sum(1)
    u = (L * B2.T[k]).sum(1) / den
    v = (L * B1.T[k]).sum(1) / den
    return t_out, k, u, v


def _exact_pixels(cam):
    """FP64 camera rays at integer pixel coordinates, row-major."""
    W, H = (int(x) for x in cam["resolution"])
    sx, sy = W / cam["sensor_size"][0], H / cam["sensor_size"][1]
    x = (torch.arange(W, dtype=torch.float64, device="cuda") - W / 2) / sx
    y = (H / 2 - torch.arange(H, dtype=torch.float64, device="cuda")) / sy
    d = torch.stack([x[None].expand(H, W), y[:, None].expand(H, W),
                     torch.full((H, W), -float(cam["focal_length"]), dtype=torch.float64, device="cuda")], -1)
    d = d.reshape(-1, 3) @ torch.as_tensor(np.asarray(cam["rotation"], np.float64)).cuda()
    d = d / d.norm(dim=1, keepdim=True)
    o = torch.as_tensor(np.asarray(cam["position"], np.float64)).cuda().expand_as(d)
    return o, d


def _exact_rays(case, q):
    P, _, _ = _triangles(q["entities"])
    r = torch.from_numpy(q["rays"]).cuda().double()
    t, _, u, v = _first_hit(P, r[:, 0:3], r[:, 4:7])
    hit = torch.isfinite(t)
    out = torch.stack([t, u, v], 1)
    return [torch.where(hit[:, None], out, 0.0), None]


def _exact_passes(case, q):
    P, N, E = _triangles(q["entities"])
    o, d = _exact_pixels(q["camera"])
    t, k, u, v = _first_hit(P, o, d)
    hit = torch.isfinite(t)[:, None]
    shape = (case["height"], case["width"], 3)
    n = torch.linalg.cross(P[k, 0] - P[k, 1], P[k, 2] - P[k, 0])
    if q["entities"][0].smooth:
        n = u[:, None] * N[k, 1] + v[:, None] * N[k, 2] + (1 - u - v)[:, None] * N[k, 0]
    n = n / n.norm(dim=1, keepdim=True)
    x = o + torch.where(hit, t[:, None], 0.0) * d
    return [torch.where(hit, x, 0.0).reshape(shape), None, torch.where(hit, n, 0.0).reshape(shape)]


def _exact_lidar(case, q):
    P, _, _ = _triangles(q["entities"])
    s = q["scan"]
    tx = torch.tan(-s["half_x"] + (torch.arange(s["nx"], dtype=torch.float64, device="cuda") + 0.5) * 2 * s["half_x"] / s["nx"])
    ty = torch.tan(-s["half_y"] + (torch.arange(s["ny"], dtype=torch.float64, device="cuda") + 0.5) * 2 * s["half_y"] / s["ny"])
    d = torch.stack([tx[None].expand(s["ny"], s["nx"]), ty[:, None].expand(s["ny"], s["nx"]),
                     -torch.ones((s["ny"], s["nx"]), dtype=torch.float64, device="cuda")], -1).reshape(-1, 3)
    d = d @ torch.as_tensor(np.asarray(s["rotation"], np.float64)).cuda()
    d = d / d.norm(dim=1, keepdim=True)
    o = torch.as_tensor(np.asarray(s["position"], np.float64)).cuda().expand_as(d)
    t, _, _, _ = _first_hit(P, o, d)
    return [torch.where(torch.isfinite(t), t, 0.0).reshape(s["ny"], s["nx"]), None]


def _exact_render(case, q):
    """Direct light of one point light at the pixel corners (one sample, one bounce): 2 pi times
    colour x (-L . n) x intensity / distance^2, where the light is not hidden."""
    P, _, E = _triangles(q["entities"])
    o, d = _exact_pixels(q["camera"])
    t, k, u, v = _first_hit(P, o, d)
    hit = torch.isfinite(t)
    n = torch.linalg.cross(P[k, 0] - P[k, 1], P[k, 2] - P[k, 0])
    n = n / n.norm(dim=1, keepdim=True)
    x = o + torch.where(hit, t, 0.0)[:, None] * d - 1e-4 * n
    light = q["lights"][0]
    to = torch.as_tensor(np.asarray(light["position"], np.float64)).cuda() - x
    dist = to.norm(dim=1, keepdim=True)
    to = to / dist
    at = torch.nonzero(hit).flatten()
    ts, _, _, _ = _first_hit(P, x[at], to[at])
    lit = torch.zeros_like(hit)
    lit[at] = ~(ts <= dist[at, 0])
    col = torch.tensor([e.color for e in q["entities"]], dtype=torch.float64, device="cuda")[E[k]]
    c = 2 * math.pi * col * (-(to * n).sum(1, keepdim=True)) * (light["intensity"] / dist ** 2).clamp(max=10000.0)
    c = torch.where((hit & lit)[:, None], c, 0.0)
    img = torch.cat([c, torch.ones_like(c[:, :1])], 1).reshape(case["height"], case["width"], 4)
    return [None, img]


def _exact_srp(case, q):
    """Flat-plate force and torque of the sun-ray grid with its specular continuations."""
    P, _, E = _triangles(q["entities"])
    s = q["srp"]
    flux, c = 1361.0, 299792458.0
    lo, hi = P.reshape(-1, 3).min(0).values, P.reshape(-1, 3).max(0).values
    ctr, Rb = 0.5 * (lo + hi), 0.5 * (hi - lo).norm()
    G = s["grid"]
    h = 2.0 * Rb / G
    rs = torch.tensor([e.rho_s for e in q["entities"]], dtype=torch.float64, device="cuda")[E]
    rd = torch.tensor([e.rho_d for e in q["entities"]], dtype=torch.float64, device="cuda")[E]
    cm = torch.tensor(s["center_of_mass"], dtype=torch.float64, device="cuda")
    F, T = [], []
    for quat in s["quaternions"]:
        R = torch.as_tensor(scenes.quaternion_to_matrix(quat / np.linalg.norm(quat))).cuda()
        sb = R.T @ torch.as_tensor(np.asarray(s["sun_dir"]) / np.linalg.norm(s["sun_dir"])).cuda()
        ax = torch.tensor([1.0, 0, 0] if abs(float(sb[0])) < 0.9 else [0, 1.0, 0], dtype=torch.float64, device="cuda")
        e1 = torch.linalg.cross(sb, ax)
        e1 = e1 / e1.norm()
        e2 = torch.linalg.cross(sb, e1)
        k = (torch.arange(G, dtype=torch.float64, device="cuda") + 0.5) * h - Rb
        o = (ctr + sb * (2 * Rb + 1) + k[:, None, None] * e2 + k[None, :, None] * e1).reshape(-1, 3)
        d = (-sb).expand_as(o)
        E_ray = (flux * h * h).expand(o.shape[0])
        f = torch.zeros(3, dtype=torch.float64, device="cuda")
        tq = torch.zeros_like(f)
        skip = None
        for seg in range(s["num_bounces"] + 1):
            t, tri, _, _ = _first_hit(P, o, d, skip)
            m = torch.nonzero(torch.isfinite(t)).flatten()
            if not len(m):
                break
            tri, d, Em = tri[m], d[m], E_ray[m]
            x = o[m] + t[m, None] * d
            n = -torch.linalg.cross(P[tri, 0] - P[tri, 1], P[tri, 2] - P[tri, 0])
            n = n / n.norm(dim=1, keepdim=True)
            n = torch.where((d * n).sum(1, keepdim=True) > 0, -n, n)
            cs = -(d * n).sum(1, keepdim=True)
            a, b = rs[tri][:, None], rd[tri][:, None]
            dF = (Em[:, None] / c) * ((1 - a) * d - (2 * a * cs + 2.0 / 3.0 * b) * n)
            f += dF.sum(0)
            tq += torch.linalg.cross(x - cm, dF).sum(0)
            go = rs[tri] > 0
            o, d, skip = (x + 1e-6 * n)[go], (d + 2 * cs * n)[go], tri[go]
            E_ray = (Em * rs[tri])[go]
        F.append(f)
        T.append(tq)
    return [torch.stack(F), torch.stack(T), None]


def exact(case, seed):
    kind, faces = case["kind"], case["faces"]
    # testing every pair takes about 20 seconds for 4e10 pairs
    if kind == "closest":
        rays = case["n"]
    elif kind in ("passes", "rebuild"):
        rays = case["width"] * case["height"]
    elif kind == "lidar":
        rays = case["nx"] * case["ny"]
    elif kind == "render" and case["spp"] == 1 and case["bounces"] == 1 and case["body"] != "cornell":
        rays = 2 * case["width"] * case["height"]
    elif kind == "srp" and case["grid"] <= 256:
        rays = 2 * case["n_att"] * case["grid"] ** 2
    else:   # whole numbers only, or sampled light: no value in 64 bits
        return None
    if rays * faces > 2e10:
        return None
    q = _request(case, seed)
    f = dict(closest=_exact_rays, passes=_exact_passes, rebuild=_exact_passes, lidar=_exact_lidar,
             render=_exact_render, srp=_exact_srp)[kind]
    return f(case, q)
