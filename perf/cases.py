"""Timed workloads of shinobi_b200, through its Python entry points.

listed() names the workloads, draw(rng) gives another one of the same ranges,
prepare(case, seed) makes what a program holds before the call (scenes, grids,
rays, request buffers), run(state) is one pass and returns its outputs,
work(case) counts the bytes and operations a pass cannot do without and
exact(case, seed) evaluates the small ones by brute force in float64.

A case's "kind" is one of

query      arbitrary rays against a resident grid (closest or any hit)
rebuild    new vertices, a grid build, then a set of probe rays
frame      a grid build and a camera frame, with ambient occlusion if ao > 0
direct     a camera frame shaded by an area light, the grid resident
dynamic    two frames of the dynamic engine (rebuild overlapped with render)
pathtrace  a path-traced image, the grid resident
batch      many scenes built and traced by one graph replay
serve      a burst of ray requests and one scene replacement on the server

Scenes: "soup" has centres U[0,1]^3 and vertex offsets U[-s,s]^3 with s scaled
so that a triangle keeps its size relative to the mean spacing of the
65,536-triangle soup (s = 0.01); "cluster" has 90% of the triangles in a ball
of radius 0.05 about the origin and 10% over [-50,50]^3; "heightfield" is a
Perlin heightfield over [0,1]^2 with boxes on it.
"""
import math

import numpy as np
import torch

import shinobi_b200 as shn
from shinobi_b200 import scenes

DEV = "cuda"
FAR = 8.0  # length of the probe rays: past every scene of unit size


def listed():
    return [
        # a tool that picks or probes: one small ray set per call, latency counts
        {"name": "query_1k", "kind": "query", "scene": "soup", "grid": "uniform", "tris": 65536, "rays": 1021,
         "any": False},
        # visibility segments in a dense cluster, the default two-level grid
        {"name": "query_any_two_level", "kind": "query", "scene": "cluster", "grid": "two_level", "tris": 262144,
         "rays": 500009, "any": True},
        # bulk ray casting (simulation, baking): millions of incoherent rays
        {"name": "query_4m", "kind": "query", "scene": "soup", "grid": "uniform", "tris": 1048576, "rays": 4000037,
         "any": False},
        # the plain uniform-grid frame: rebuild and 512 x 512 primary rays
        {"name": "frame_soup", "kind": "frame", "scene": "soup", "grid": "uniform", "insertion": "plane",
         "tris": 65536, "width": 512, "height": 512, "ao": 0},
        # the same size with the precise insertion rule and an odd image
        {"name": "frame_soup_sat", "kind": "frame", "scene": "soup", "grid": "uniform", "insertion": "sat",
         "tris": 99991, "width": 401, "height": 307, "ao": 1},
        # the headline frame: two-level rebuild, 1920 x 1080 primary, 4 AO rays per hit
        {"name": "frame_cluster_1080p", "kind": "frame", "scene": "cluster", "grid": "two_level_flat",
         "insertion": "plane", "tris": 1048576, "width": 1920, "height": 1080, "ao": 4},
        # static geometry under a moving camera: primary rays and area-light shading
        {"name": "direct_cluster", "kind": "direct", "scene": "cluster", "grid": "two_level_flat", "tris": 524287,
         "width": 1283, "height": 717, "samples": 4},
        # animation: interpolated vertices, rebuild overlapped with the render
        {"name": "dynamic_cluster", "kind": "dynamic", "scene": "cluster", "grid": "two_level_flat", "tris": 262144,
         "width": 960, "height": 540, "samples": 4},
        # a large scene whose vertices changed: the build is the work
        {"name": "rebuild_4m", "kind": "rebuild", "scene": "soup", "grid": "uniform", "tris": 4194304, "rays": 65536},
        # the large path-traced scene: 4.2M triangles, 1920 x 1080 x 16 paths, depth 4
        {"name": "pathtrace_1080p", "kind": "pathtrace", "scene": "heightfield", "grid": "uniform", "quads_x": 2048,
         "quads_y": 1024, "boxes": 1000, "width": 1920, "height": 1080, "spp": 16, "depth": 4},
        # many scenes of uneven size in one captured step
        {"name": "batch_64", "kind": "batch", "scenes": 64, "tris_max": 524288, "rays_max": 262144},
        # a burst of requests for resident scenes, host memory to host memory
        {"name": "serve_256", "kind": "serve", "scenes": 8, "tris": 131072, "requests": 256, "rays_max": 65536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "frame", "frame", "direct", "dynamic", "rebuild", "pathtrace", "batch",
                       "serve"])
    grid = rng.choice(["uniform", "two_level", "two_level_flat"])
    # cells of equal size suit evenly spread triangles, two levels suit a cluster
    scene = "soup" if grid == "uniform" else rng.choice(["cluster", "cluster", "soup"])
    if kind == "query":
        return {"kind": kind, "scene": scene, "grid": grid, "tris": _log(rng, 4096, 1 << 20),
                "rays": _log(rng, 512, 4000000), "any": rng.random() < 0.5}
    if kind == "rebuild":
        return {"kind": kind, "scene": scene, "grid": grid, "tris": _log(rng, 16384, 1 << 22),
                "rays": _log(rng, 4096, 65536)}
    w = _log(rng, 160, 1920)
    h = max(90, min(1080, int(w * rng.uniform(0.5, 0.8))))
    if kind == "frame":
        return {"kind": kind, "scene": scene, "grid": grid,
                "insertion": rng.choice(["plane", "plane", "sat"]) if grid == "uniform" else "plane",
                "tris": _log(rng, 16384, 1 << 20), "width": w, "height": h, "ao": rng.choice([0, 1, 2, 4])}
    if kind in ("direct", "dynamic"):
        return {"kind": kind, "scene": "cluster", "grid": rng.choice(["two_level", "two_level_flat"]),
                "tris": _log(rng, 32768, 1 << 20), "width": w, "height": h, "samples": rng.choice([1, 2, 4])}
    if kind == "pathtrace":
        q = _log(rng, 128, 1024)
        return {"kind": kind, "scene": "heightfield", "grid": rng.choice(["uniform", "uniform", "two_level"]),
                "quads_x": q, "quads_y": q // 2 + 1, "boxes": _log(rng, 10, 500), "width": w, "height": h,
                "spp": rng.choice([1, 2, 4, 8]), "depth": rng.choice([2, 3, 4, 6])}
    if kind == "batch":
        return {"kind": kind, "scenes": _log(rng, 8, 64), "tris_max": _log(rng, 32768, 524288),
                "rays_max": _log(rng, 32768, 262144)}
    return {"kind": kind, "scenes": rng.randint(2, 8), "tris": _log(rng, 16384, 131072),
            "requests": _log(rng, 32, 256), "rays_max": _log(rng, 8192, 65536)}


# ---- inputs -------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (1 << 62) + 1)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float32)


def _unit(g, n):
    z = 2.0 * _rand(g, n).double() - 1.0
    phi = 2.0 * math.pi * _rand(g, n).double()
    rho = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
    return torch.stack([rho * torch.cos(phi), rho * torch.sin(phi), z], dim=1)


def _faces(n):
    return torch.arange(3 * n, dtype=torch.int32, device=DEV).reshape(n, 3)


def _soup(g, n):
    s = 0.01 * (65536.0 / n) ** (1.0 / 3.0)
    c = _rand(g, n, 1, 3)
    return (c + (2.0 * _rand(g, n, 3, 3) - 1.0) * s).reshape(3 * n, 3).contiguous()


def _cluster(g, n):
    nc = int(round(0.9 * n))
    r = 0.05 * _rand(g, nc, 1).double() ** (1.0 / 3.0)
    c = (_unit(g, nc) * r).float()
    a = c[:, None, :] + (2.0 * _rand(g, nc, 3, 3) - 1.0) * 0.002
    f = (2.0 * _rand(g, n - nc, 1, 3) - 1.0) * 50.0
    b = f + (2.0 * _rand(g, n - nc, 3, 3) - 1.0) * 0.5
    return torch.cat([a, b]).reshape(3 * n, 3).contiguous()


def _perlin(g, x, y, octaves=4):
    """Sum of `octaves` octaves of 2D gradient noise at (x, y) in [0, 1]^2."""
    ang = 2.0 * math.pi * _rand(g, 128, 128).double()
    gx, gy = torch.cos(ang), torch.sin(ang)
    z = torch.zeros_like(x)
    freq, amp = 4.0, 1.0
    for _ in range(octaves):
        px, py = x * freq, y * freq
        ix, iy = px.floor().long(), py.floor().long()
        fx, fy = px - ix, py - iy
        u, v = (t * t * t * (t * (t * 6 - 15) + 10) for t in (fx, fy))

        def corner(dx, dy):
            j, i = (iy + dy) & 127, (ix + dx) & 127
            return gx[j, i] * (fx - dx) + gy[j, i] * (fy - dy)

        top = corner(0, 0) * (1 - u) + corner(1, 0) * u
        bot = corner(0, 1) * (1 - u) + corner(1, 1) * u
        z = z + amp * (top * (1 - v) + bot * v)
        freq, amp = freq * 2.0, amp * 0.5
    return z


def _heightfield(g, w, h, boxes):
    state = g.get_state()
    y, x = torch.meshgrid(torch.linspace(0, 1, h + 1, device=DEV, dtype=torch.float64),
                          torch.linspace(0, 1, w + 1, device=DEV, dtype=torch.float64), indexing="ij")
    z = 0.1 * _perlin(g, x, y)
    hv = torch.stack([x, y, z], dim=-1).reshape(-1, 3).float()
    j, i = torch.meshgrid(torch.arange(h, device=DEV), torch.arange(w, device=DEV), indexing="ij")
    a = (j * (w + 1) + i).reshape(-1)
    b, c, d = a + 1, a + w + 1, a + w + 2
    hi = torch.stack([torch.stack([a, b, d], 1), torch.stack([a, d, c], 1)], 1).reshape(-1, 3)
    xy = _rand(g, boxes, 2).double()
    side = torch.exp(-4.0 + 0.5 * torch.randn(boxes, generator=g, device=DEV, dtype=torch.float32).double())
    again = torch.Generator(device=DEV)
    again.set_state(state)
    bz = 0.1 * _perlin(again, xy[:, 0].contiguous(), xy[:, 1].contiguous())
    lo = torch.stack([xy[:, 0] - side / 2, xy[:, 1] - side / 2, bz - side / 4], 1)
    k = torch.arange(8, device=DEV)
    corner = torch.stack([k & 1, (k >> 1) & 1, (k >> 2) & 1], 1).double()
    bv = (lo[:, None] + corner[None] * side[:, None, None]).reshape(-1, 3).float()
    tri = torch.tensor([[0, 2, 1], [1, 2, 3], [4, 5, 6], [5, 7, 6], [0, 1, 4], [1, 5, 4],
                        [2, 6, 3], [3, 6, 7], [0, 4, 2], [2, 4, 6], [1, 3, 5], [3, 7, 5]], device=DEV)
    bi = (hv.shape[0] + 8 * torch.arange(boxes, device=DEV)[:, None, None] + tri[None]).reshape(-1, 3)
    return torch.cat([hv, bv]).contiguous(), torch.cat([hi, bi]).to(torch.int32).contiguous()


def _triangles(c, g):
    if c["scene"] == "heightfield":
        return _heightfield(g, c["quads_x"], c["quads_y"], c["boxes"])
    v = _soup(g, c["tris"]) if c["scene"] == "soup" else _cluster(g, c["tris"])
    return v, _faces(c["tris"])


def _params(c):
    insertion = shn.SHN_INSERT_SAT if c.get("insertion") == "sat" else shn.SHN_INSERT_PLANE
    if c["grid"] == "uniform":
        return shn.grid_params(shn.SHN_GRID_UNIFORM, insertion=insertion)
    if c["grid"] == "two_level":
        return shn.grid_params(shn.SHN_GRID_TWO_LEVEL, insertion=insertion)
    # few top cells over a sparse field, dense leaves in the cluster
    return shn.grid_params(shn.SHN_GRID_TWO_LEVEL, lambda_=1.0 / 16.0, top_divisor=1, min_res=2, lambda_leaf=4.0,
                           leaf_threshold=16, insertion=insertion)


def _rays(c, g):
    """Origins, directions, lengths.  Any-hit segments are short, as occlusion queries are."""
    n = c["rays"]
    if c["scene"] == "cluster":
        org = (2.0 * _rand(g, n, 3) - 1.0) * 0.15
        length = 0.1 if c.get("any") else 200.0
    else:
        org = 3.0 * _rand(g, n, 3) - 1.0
        length = 0.5 if c.get("any") else FAR
    return org.contiguous(), _unit(g, n).float().contiguous(), torch.full((n,), length, device=DEV)


def _camera(c):
    base = {"soup": scenes.CAMERA_SOUP, "cluster": scenes.CAMERA_CLUSTER,
            "heightfield": scenes.CAMERA_HEIGHTFIELD}[c["scene"]]
    return scenes.Camera(base.eye, base.forward, base.up, base.fov_deg, c["width"], c["height"])


def _sizes(c, seed, lo, hi, n, salt):
    r = np.random.RandomState((int(seed) * 7919 + salt) % (1 << 31))
    return np.exp(r.uniform(math.log(lo), math.log(hi), n)).astype(np.int64), r


class _HostScene:
    def __init__(self, v, i):
        self.vertices, self.indices = v, i


def _prepare_batch(c, seed, g):
    # one size distribution per case: the seed moves the geometry, not the amount of work
    tris, r = _sizes(c, 3, 1000, c["tris_max"], c["scenes"], 1)
    scale = np.exp(r.uniform(math.log(0.001), math.log(0.05), c["scenes"]))
    rays, _ = _sizes(c, 3, max(1024, c["rays_max"] // 16), c["rays_max"], c["scenes"], 2)
    hosts = []
    for n, s in zip(tris.tolist(), scale.tolist()):
        v = (_rand(g, n, 1, 3) + (2.0 * _rand(g, n, 3, 3) - 1.0) * s).reshape(3 * n, 3)
        hosts.append(_HostScene(v.cpu().numpy(), np.arange(3 * n, dtype=np.uint32).reshape(n, 3)))
    off = np.concatenate([[0], np.cumsum(rays)]).astype(np.uint32)
    n = int(off[-1])
    org = (3.0 * _rand(g, n, 3) - 1.0).contiguous()
    d = _unit(g, n).float().contiguous()
    b = shn.Batch(hosts)
    out = shn.alloc_hits(n)
    b.capture(org, d, off, out)
    return {"kind": "batch", "batch": b, "out": out}


def _prepare_serve(c, seed, g):
    sv = shn.Server(num_slots=c["scenes"])
    fresh = None
    for s in range(c["scenes"]):
        n = max(1000, c["tris"] >> (s % 4))
        host = _HostScene(_soup(g, n).cpu().numpy(), np.arange(3 * n, dtype=np.uint32).reshape(n, 3))
        sv.load_scene(s, host)
        if s == 0:
            fresh = _HostScene(_soup(g, n).cpu().numpy(), host.indices)
    rays, r = _sizes(c, 5, 1024, c["rays_max"], c["requests"], 3)
    slot = r.randint(0, c["scenes"], c["requests"])
    slot = slot[np.argsort(slot == 0, kind="stable")]  # the replaced scene is asked for after its replacement
    anyhit = r.rand(c["requests"]) < 0.5
    total = int(rays.sum())
    rec = torch.empty(total, 8, dtype=torch.float32, device=DEV)
    rec[:, 0:3] = 3.0 * _rand(g, total, 3) - 1.0
    rec[:, 3:6] = _unit(g, total).float()
    rec[:, 6] = FAR
    rec[:, 7] = 0.0
    host = torch.empty(total, 8, dtype=torch.float32, pin_memory=True)
    host.copy_(rec)
    tri = torch.zeros(total, dtype=torch.int32, pin_memory=True)
    t = torch.zeros(total, dtype=torch.float32, pin_memory=True)
    reqs, at = [sv.update_request(0, fresh)], 0
    for n, s, a in zip(rays.tolist(), slot.tolist(), anyhit.tolist()):
        reqs.append(sv.ray_request(shn._abi.SHN_REQ_ANY if a else shn._abi.SHN_REQ_CLOSEST, s, host[at:at + n],
                                   tri[at:at + n], t[at:at + n]))
        at += n
    return {"kind": "serve", "server": sv, "reqs": reqs, "arrival": np.zeros(len(reqs)), "host": host, "tri": tri,
            "t": t, "fresh": fresh}


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed, g)
    if kind == "serve":
        return _prepare_serve(case, seed, g)
    v, f = _triangles(case, g)
    p = _params(case)
    s = {"kind": kind, "params": p, "ao": case.get("ao", 0)}
    if kind in ("frame", "direct", "dynamic", "pathtrace"):
        s["cam"] = _camera(case)
    if kind == "dynamic":
        s["kf"] = [v, (v + 0.001 * (2.0 * _rand(g, *v.shape) - 1.0)).contiguous()]
        s["engine"] = shn.DynamicEngine(v, f, p)
        n = case["width"] * case["height"]
        s["hits"] = [shn.alloc_hits(n) for _ in range(2)]
        s["frames"] = [torch.empty(case["height"], case["width"], 3, device=DEV) for _ in range(2)]
        s["di"] = shn.di_params(samples=case["samples"])
        return s
    s["soup"] = shn.FaceSoup(v, f)
    s["grid"] = shn.Grid()
    if kind == "rebuild":
        s["vertices"] = v
    if kind in ("query", "rebuild"):
        s["rays"] = _rays(case, g)
    if kind in ("query", "direct", "pathtrace"):
        s["grid"].build(s["soup"], p)
    if kind == "query":
        s["any"] = case["any"]
    if kind == "direct":
        s["di"] = shn.di_params(samples=case["samples"])
    if kind == "pathtrace":
        s["pt"] = shn.pt_params(spp=case["spp"], max_depth=case["depth"])
    return s


# ---- one pass -----------------------------------------------------------------------
def _hits(h):
    return {"tri": h.tri, "t": h.t, "u": h.u, "v": h.v}


def run(state):
    s = state
    kind = s["kind"]
    if kind == "query":
        if s["any"]:
            return s["grid"].trace_any(*s["rays"])
        return _hits(s["grid"].trace_closest(*s["rays"]))
    if kind == "rebuild":
        s["soup"].update_vertices(s["vertices"])
        s["grid"].build(s["soup"], s["params"])
        return _hits(s["grid"].trace_closest(*s["rays"]))
    if kind == "frame":
        s["grid"].build(s["soup"], s["params"])
        h = s["grid"].trace_primary(s["cam"])
        out = _hits(h)
        if s["ao"]:
            out["ao"] = s["grid"].trace_ao(s["cam"], h, spp=s["ao"], length=0.1, offset=1e-4, seed=1)
        return out
    if kind == "direct":
        h = s["grid"].trace_primary(s["cam"])
        return dict(_hits(h), frame=s["grid"].shade_direct(s["cam"], h, s["di"]))
    if kind == "dynamic":
        for k, coeff in enumerate((0.25, 0.75)):
            s["engine"].render_frame(s["kf"][0], s["kf"][1], coeff, s["cam"], s["di"], s["hits"][k], s["frames"][k])
        # the second frame shows the first call's geometry, whatever was rendered before
        return dict(_hits(s["hits"][1]), frame=s["frames"][1])
    if kind == "pathtrace":
        return s["grid"].pt_render(s["soup"], s["cam"], s["pt"])
    if kind == "batch":
        s["batch"].replay()
        return _hits(s["out"])
    s["server"].run_schedule(s["reqs"], s["arrival"])
    return {"tri": s["tri"], "t": s["t"]}


# ---- what a pass cannot do without --------------------------------------------------
HIT = 16   # tri, t, u, v
RAY = 28   # origin, direction, length
TRI = 36   # three vertices
TEST = 40  # operations of one ray/triangle test; a ray needs at least one


def work(case):
    c = case
    kind = c["kind"]
    if kind == "query":
        n = c["rays"]
        return {"bytes": TRI * c["tris"] + n * (RAY + (1 if c["any"] else HIT)), "flops": TEST * n}
    if kind == "rebuild":
        return {"bytes": (TRI + 12) * c["tris"] + c["rays"] * (RAY + HIT), "flops": TEST * c["rays"]}
    if kind == "batch":
        tris = int(_sizes(c, 3, 1000, c["tris_max"], c["scenes"], 1)[0].sum())
        rays = int(_sizes(c, 3, max(1024, c["rays_max"] // 16), c["rays_max"], c["scenes"], 2)[0].sum())
        return {"bytes": (TRI + 12) * tris + rays * (24 + HIT), "flops": TEST * rays}
    if kind == "serve":
        rays = int(_sizes(c, 5, 1024, c["rays_max"], c["requests"], 3)[0].sum())
        return {"bytes": (TRI + 12) * c["tris"] + rays * (32 + 8), "flops": TEST * rays}
    tris = 2 * c["quads_x"] * c["quads_y"] + 12 * c["boxes"] if kind == "pathtrace" else c["tris"]
    n = c["width"] * c["height"]
    if kind == "frame":
        return {"bytes": (TRI + 12) * tris + n * (HIT + (4 if c["ao"] else 0)), "flops": TEST * n * (1 + c["ao"])}
    if kind == "direct":
        return {"bytes": TRI * tris + n * (HIT + 12), "flops": TEST * n * (1 + c["samples"])}
    if kind == "dynamic":
        return {"bytes": 2 * (2 * TRI * tris + n * (HIT + 12)), "flops": 2 * TEST * n * (1 + c["samples"])}
    return {"bytes": TRI * tris + 12 * n, "flops": TEST * n * c["spp"] * 2}


# ---- float64 values of the small cases ----------------------------------------------
def _brute(v, org, d, tmax, miss):
    """Closest hits of rays against all triangles (Moller-Trumbore in float64): t, u, v."""
    a, b, c = (x.double() for x in v.reshape(-1, 3, 3).unbind(1))
    e1, e2 = b - a, c - a
    nrm = torch.linalg.cross(e1, e2)
    n = org.shape[0]
    out = [torch.empty(n, dtype=torch.float64, device=DEV) for _ in range(3)]
    step = max(1, (1 << 27) // max(1, a.shape[0]))
    for i in range(0, n, step):
        o, w = org[i:i + step].double(), d[i:i + step].double()
        # det = -d . n;  t = (o - a) . n / det;  u, v from q = (o - a) x d
        det = -(w @ nrm.T)
        t = (o @ nrm.T - (a * nrm).sum(1)) / det
        m = torch.linalg.cross(o, w)  # q = o x d - a x d
        # e2 . (a x d) = d . (e2 x a), and so for e1
        qu = m @ e2.T - w @ torch.linalg.cross(e2, a).T
        u = qu / det
        qv = m @ e1.T - w @ torch.linalg.cross(e1, a).T
        w2 = -qv / det
        ok = (u >= 0) & (w2 >= 0) & (u + w2 <= 1) & (t > 1e-5) & (t < tmax[i:i + step].double()[:, None])
        t = torch.where(ok, t, math.inf)
        best, k = t.min(1)
        hit = torch.isfinite(best)
        r = torch.arange(o.shape[0], device=DEV)
        out[0][i:i + step] = torch.where(hit, best, miss)
        out[1][i:i + step] = torch.where(hit, u[r, k], 0.0)
        out[2][i:i + step] = torch.where(hit, w2[r, k], 0.0)
    return out


def _camera_rays(cam):
    """Directions through the pixel centres, float64."""
    f, up = (torch.tensor(x, dtype=torch.float64) for x in (cam.forward, cam.up))
    f = f / f.norm()
    r = torch.linalg.cross(f, up)
    r = r / r.norm()
    u = torch.linalg.cross(f, r)
    u = u / u.norm()
    tn = math.tan(math.radians(cam.fov_deg) / 2.0)
    row, col = r * 2.0 * tn * cam.res_x / cam.res_y, u * 2.0 * tn
    y, x = torch.meshgrid(torch.arange(cam.res_y, dtype=torch.float64) + 0.5,
                          torch.arange(cam.res_x, dtype=torch.float64) + 0.5, indexing="ij")
    d = f + (x.reshape(-1, 1) / cam.res_x - 0.5) * row + (y.reshape(-1, 1) / cam.res_y - 0.5) * col
    return d.to(DEV).contiguous()


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("query", "rebuild", "frame") or case.get("any"):
        return None
    rays = case["width"] * case["height"] if kind == "frame" else case["rays"]
    if rays * case["tris"] > 4e10:
        return None
    g = _gen(seed)
    v, _ = _triangles(case, g)
    if kind == "frame":
        cam = _camera(case)
        d = _camera_rays(cam)
        org = torch.tensor(cam.eye, dtype=torch.float64, device=DEV).expand(rays, 3)
        far = torch.full((rays,), math.inf, dtype=torch.float64, device=DEV)
        t, u, w = _brute(v, org, d, far, float(np.finfo(np.float32).max))
    else:
        org, d, far = _rays(case, g)
        t, u, w = _brute(v, org, d, far, float(far[0]))
    out = {"tri": None, "t": t, "u": u, "v": w}
    if case.get("ao"):
        out["ao"] = None
    return out
