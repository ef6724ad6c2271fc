"""Uniform-grid traversal at the edges of the flat engine: ray counts around a
warp, one-cell axes, ranges beyond the shared-load limit, start cells outside
the grid, axis-parallel, degenerate and non-finite rays.

Every result is compared bit for bit with the one-ray-per-lane engine (which
the counting variant of the kernels runs), and with the oracle for the rays
whose floats are all finite.
"""
import numpy as np
import pytest

import oracle
from shinobi_b200 import scenes

pytestmark = pytest.mark.gpu


def _rays(n, b, seed):
    r = np.random.RandomState(seed)
    lo, hi = b[:3], b[3:]
    ext = hi - lo
    org = (lo + ext * r.uniform(-1.0, 2.0, (n, 3))).astype(np.float32)
    d = r.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    k = np.arange(n)
    org[k % 7 == 1] = (lo + ext * r.uniform(0.05, 0.95, (n, 3)))[k % 7 == 1]      # inside
    far = k % 7 == 2                                                               # start cells off by rounding
    aim = (lo + ext * r.uniform(0.1, 0.9, (n, 3)))
    org[far] = (aim - d * (10.0 ** r.uniform(2, 7, (n, 1))) * ext.max())[far]
    d[k % 7 == 3, 0] = 0.0                                                         # parallel to a plane
    axis = k % 7 == 4                                                              # parallel to an axis
    d[axis] = 0.0
    d[axis, k[axis] % 3] = np.where(r.rand(int(axis.sum())) < 0.5, 1.0, -1.0)
    face = k % 21 == 5                                                             # origin on a face of the box
    org[face, 2] = lo[2]
    tmax = np.where(k % 5 == 0, r.uniform(0.0, 1.0, n) * ext.max(), 3.0e38).astype(np.float32)
    tmax[k % 31 == 7] = 0.0
    return org, d, tmax


@pytest.mark.parametrize("tris,scale,res,rays", [
    (1, 0.3, (1, 1, 1), 1),
    (5, 0.5, (3, 1, 2), 31),
    (300, 0.05, (7, 7, 7), 33),
    (3000, 0.02, (1, 40, 3), 1000),       # up to ~100 references in a cell
    (20000, 0.01, (2, 2, 2), 777),        # thousands of references in a cell
    (20000, 0.01, (40, 41, 39), 20011),
    (20000, 0.01, (40, 41, 39), 131071),  # either side of the window lengths' limit
    (20000, 0.01, (40, 41, 39), 131072),
    (40000, 0.004, (163, 162, 161), 30001),  # above the size with empty-cell distances
    (2000, 0.01, (2048, 2, 3), 5003),     # the longest axis
])
def test_flat_traversal(gpu, tris, scale, res, rays):
    import torch

    import shinobi_b200 as shn
    sc = scenes.uniform_soup(tris, seed=tris, offset_scale=scale)
    soup = shn.FaceSoup(sc.vertices, sc.indices)
    g = shn.Grid().build(soup, shn.grid_params(shn.SHN_GRID_UNIFORM, res=res))
    b = oracle.bounds(sc.vertices, sc.indices)
    org, d, tmax = _rays(rays, b, seed=rays)
    odd = np.arange(rays) % 97 == 11  # not finite
    org[odd, 0] = np.nan
    d[odd & (np.arange(rays) % 2 == 0), 1] = np.inf
    dev = [torch.from_numpy(x).cuda() for x in (org, d, tmax)]
    h = g.trace_closest(*dev)
    occ = g.trace_any(*dev)
    plain = shn.alloc_hits(rays, uv=False)
    g.trace_closest(*dev, out=plain)
    cnt = torch.zeros(2, dtype=torch.int64, device="cuda")
    shn.default_context().lib.shn_grid_set_stats(g.handle, shn._ptr(cnt))
    try:
        h2 = g.trace_closest(*dev)
        occ2 = g.trace_any(*dev)
    finally:
        shn.default_context().lib.shn_grid_set_stats(g.handle, None)
    torch.cuda.synchronize()
    bits = [np.ascontiguousarray(x.cpu().numpy()).view(np.uint32) for x in (h.tri, h.t, h.u, h.v)]
    for name, a, x in zip(("tri", "t", "u", "v"), bits, (h2.tri, h2.t, h2.u, h2.v)):
        assert np.array_equal(a, x.cpu().numpy().view(np.uint32)), f"{name} differs from the per-lane engine"
    assert torch.equal(occ, occ2)
    assert torch.equal(plain.tri, h.tri) and torch.equal(plain.t.view(torch.int32), h.t.view(torch.int32))
    og = oracle.build_uniform(sc.vertices, sc.indices, b, np.array(res, np.int32))
    keep = ~odd
    ref = oracle.trace_closest(og, org[keep], d[keep], tmax[keep])
    for name, a, x in zip(("tri", "t", "u", "v"), bits, ref):
        assert np.array_equal(a[keep], np.ascontiguousarray(x).view(np.uint32)), f"{name} differs from the oracle"
    ro = oracle.trace_any(og, org[keep], d[keep], tmax[keep])[0]
    assert np.array_equal(occ.cpu().numpy()[keep], np.asarray(ro).astype(np.uint8))


@pytest.mark.parametrize("kind", [0, 1])
def test_strided_rays(gpu, kind):
    """Rays read in place from sliced, transposed, repeated and padded arrays equal contiguous ones."""
    import torch

    import shinobi_b200 as shn
    sc = scenes.uniform_soup(20000, seed=3)
    g = shn.Grid().build(shn.FaceSoup(sc.vertices, sc.indices), shn.grid_params(kind))
    b = oracle.bounds(sc.vertices, sc.indices)
    org, d, tmax = [torch.from_numpy(x).cuda() for x in _rays(3001, b, seed=5)]
    n = org.shape[0]
    pad = torch.zeros(n, 8, device="cuda")
    pad[:, 1:4], pad[:, 4:7], pad[:, 7] = org, d, tmax
    one = org[1:2].expand(n, 3)
    forms = [
        (org, d, tmax, org, d, tmax),
        (pad[:, 1:4], pad[:, 4:7], pad[:, 7], org, d, tmax),
        (org.t().contiguous().t(), d.t().contiguous().t(), tmax, org, d, tmax),
        (org[::2], d[::2], tmax[::2], org[::2].contiguous(), d[::2].contiguous(), tmax[::2].contiguous()),
        (one, d, tmax[:1].expand(n), one.contiguous(), d, tmax[:1].expand(n).contiguous()),
        (org, d, None, org, d, torch.full((n,), 3.4028234663852886e38, device="cuda")),
    ]
    for o, w, t, o2, w2, t2 in forms:
        ref = shn.alloc_hits(o.shape[0])
        rays, keep = shn.Grid._rays(o2, w2, t2)
        import ctypes as C
        h = ref.struct()
        g.ctx.check(g.ctx.lib.shn_trace_closest(g.handle, C.byref(rays), o.shape[0], C.byref(h), shn._stream(None)), "")
        got = g.trace_closest(o, w, t)
        for a, x in ((got.tri, ref.tri), (got.t, ref.t), (got.u, ref.u), (got.v, ref.v)):
            assert torch.equal(a.view(torch.int32), x.view(torch.int32))
        if t is not None:
            assert torch.equal(g.trace_any(o, w, t).bool(), ref.tri != -1)


@pytest.mark.parametrize("lambdas,rays", [((5.0, 0.5, 0.004), 1501), ((0.004, 0.02), 33), ((5.0,), 1)])
def test_mixed_requests(gpu, lambdas, rays):
    """Closest- and any-hit requests of several scenes in one launch, ranges of a few to thousands of
    references: closest hits equal the oracle's bit for bit, any-hit answers its occlusion, and an any-hit
    triangle is one the ray hits at the t given."""
    import torch

    import shinobi_b200 as shn
    sv = shn.Server(num_slots=len(lambdas))
    try:
        reqs, want, keep = [], [], []
        for k, lam in enumerate(lambdas):
            sc = scenes.uniform_soup(4000 + 500 * k, seed=k + 1, offset_scale=0.02)
            sv.load_scene(k, sc, lam)
            b = oracle.bounds(sc.vertices, sc.indices)
            og = oracle.build_uniform(sc.vertices, sc.indices, b, oracle.resolution(sc.num_triangles, b, lam, 1, 1))
            for kind in (0, 1):
                org, d, tmax = _rays(rays + 7 * k, b, seed=10 * k + kind)
                r8 = torch.zeros(org.shape[0], 8).pin_memory()
                r8[:, 0:3], r8[:, 3:6], r8[:, 6] = map(torch.from_numpy, (org, d, tmax))
                tri = torch.zeros(org.shape[0], dtype=torch.int32).pin_memory()
                t = torch.zeros(org.shape[0]).pin_memory()
                reqs.append(sv.ray_request(kind, k, r8, tri, t))
                keep.append(r8)
                want.append((kind, sc, og, org, d, tmax, tri, t))
        res = sv.run_schedule(reqs, np.zeros(len(reqs)))
        assert not res.any()
        for kind, sc, og, org, d, tmax, tri, t in want:
            tri, t = tri.numpy().view(np.uint32), t.numpy()
            if kind == 0:
                rt, rtt = oracle.trace_closest(og, org, d, tmax)[:2]
                assert np.array_equal(tri, rt) and np.array_equal(t.view(np.uint32), rtt.view(np.uint32))
            else:
                occ = np.asarray(oracle.trace_any(og, org, d, tmax)[0]).astype(bool)
                hit = tri != shn.SHN_MISS
                assert np.array_equal(hit, occ)
                t64 = oracle.t_fp64(sc.vertices, sc.indices, tri, org, d)
                near = hit & (np.abs(org).max(1) < 10.0)  # distant origins: t carries their rounding
                assert np.all(np.abs(t[near] - t64[near]) <= 1e-4 * np.maximum(1.0, np.abs(t64[near])))
    finally:
        sv.close()


@pytest.mark.parametrize("counts", [
    (0, 3, 0, 100, 0, 40, 1, 0),       # short ranges before and behind long ones, a window's cells or two
    (40, 0, 33, 1, 32, 31, 200, 64),
    (1, 700, 1, 700, 1, 65, 0, 5),
    (32, 33, 63, 64, 65, 95, 96, 97),  # around the lengths at which the engine changes
])
def test_any_hit_request_answer(gpu, counts):
    """The triangle and t of an any-hit request are those of the first cell on the ray with a hit: there the
    first reference that is hit of a range of up to 32, else the nearest hit of the first 32 references
    that hold one.  Layers of triangles across the rays, sorted neither by depth nor by size."""
    import torch

    import shinobi_b200 as shn
    r = np.random.RandomState(sum(counts))
    layer = np.repeat(np.arange(8), counts)
    r.shuffle(layer)
    nt = layer.size + 8
    x = np.empty(layer.size)
    for c in range(8):  # inside the cell, 0.0004 apart or more
        k = np.flatnonzero(layer == c)
        x[k] = (c + 0.2 + 0.6 * (r.permutation(k.size) + 0.5) / max(1, k.size)) / 8.0
    ang = np.sort(r.uniform(0, 2 * np.pi, (layer.size, 3)), axis=1)
    tri = np.empty((nt, 3, 3))
    tri[8:, :, 0] = x[:, None]
    tri[8:, :, 1], tri[8:, :, 2] = 0.5 + 0.48 * np.cos(ang), 0.5 + 0.48 * np.sin(ang)
    for k in range(8):  # the corners of the unit cube, so that the cells are its eighths
        corner = np.array([k & 1, k >> 1 & 1, k >> 2 & 1], float)
        tri[k] = corner + np.array([[0, 0, 0], [1e-3, 0, 0], [0, 1e-3, 0]]) * (1 - 2 * corner)
    v = tri.reshape(-1, 3).astype(np.float32)
    sc = type("S", (), {"vertices": v, "indices": np.arange(3 * nt, dtype=np.uint32).reshape(nt, 3),
                        "num_triangles": nt})
    lam = 8.5 ** 3 / nt
    b = oracle.bounds(v, sc.indices)
    res = oracle.resolution(nt, b, lam, 1, 1)
    assert tuple(res) == (8, 8, 8) and np.allclose(b, [0, 0, 0, 1, 1, 1])
    og = oracle.build_uniform(v, sc.indices, b, res)

    n = 1500
    cy, cz = r.randint(1, 7, n), r.randint(1, 7, n)
    sign = np.where(r.rand(n) < 0.5, 1.0, -1.0)
    org = np.empty((n, 3))
    org[:, 0] = np.where(r.rand(n) < 0.7, np.where(sign > 0, -0.5, 1.5), r.uniform(0.0, 1.0, n))
    org[:, 1], org[:, 2] = (cy + r.uniform(0.3, 0.7, n)) / 8.0, (cz + r.uniform(0.3, 0.7, n)) / 8.0
    org = org.astype(np.float32)
    d = np.stack([sign, r.uniform(-1e-3, 1e-3, n), r.uniform(-1e-3, 1e-3, n)], 1).astype(np.float32)
    d[::5, 1:] = 0.0
    tmax = np.where(r.rand(n) < 0.7, 8.0, r.uniform(0.2, 1.5, n)).astype(np.float32)

    # every (ray, triangle) pair in float64; rays that pass an edge or a bound closely are left out
    a = v.reshape(nt, 3, 3).astype(np.float64)[8:]
    o64, d64 = org.astype(np.float64), d.astype(np.float64)
    t = (a[None, :, 0, 0] - o64[:, None, 0]) / d64[:, None, 0]
    p = o64[:, None, 1:] + t[..., None] * d64[:, None, 1:]
    e = []
    for k in range(3):
        s, f = a[None, :, k, 1:], a[None, :, (k + 1) % 3, 1:]
        e.append((f[..., 0] - s[..., 0]) * (p[..., 1] - s[..., 1]) - (f[..., 1] - s[..., 1]) * (p[..., 0] - s[..., 0]))
    e = np.stack(e)
    hit = (e > 0).all(0) & (t > 1e-5) & (t < tmax[:, None])
    sure = ((np.abs(e) > 1e-5).all(0) & (np.abs(t - 1e-5) > 1e-4) & (np.abs(t - tmax[:, None]) > 1e-4)).all(1)
    assert sure.sum() > n // 4

    r8 = torch.zeros(n, 8).pin_memory()
    r8[:, 0:3], r8[:, 3:6], r8[:, 6] = map(torch.from_numpy, (org, d, tmax))
    got, gt = torch.zeros(n, dtype=torch.int32).pin_memory(), torch.zeros(n).pin_memory()
    near, nt_ = torch.zeros(n, dtype=torch.int32).pin_memory(), torch.zeros(n).pin_memory()
    sv = shn.Server(num_slots=1)
    try:
        sv.load_scene(0, sc, lam)
        out = sv.run_schedule([sv.ray_request(shn._abi.SHN_REQ_ANY, 0, r8, got, gt),
                               sv.ray_request(shn._abi.SHN_REQ_CLOSEST, 0, r8, near, nt_)], np.zeros(2))
        assert not out.any()
    finally:
        sv.close()
    got, gt = got.numpy().view(np.uint32), gt.numpy()
    ref = oracle.trace_closest(og, org, d, tmax)
    assert np.array_equal(near.numpy().view(np.uint32), ref[0])
    assert np.array_equal(nt_.numpy().view(np.uint32), ref[1].view(np.uint32))
    seen = set()
    for i in np.flatnonzero(sure):
        want = shn.SHN_MISS
        for x_ in (range(8) if sign[i] > 0 else range(7, -1, -1)):
            lo, hi = og.cells[x_ + 8 * cy[i] + 64 * cz[i]]
            ids = og.indices[lo:hi].astype(np.int64) - 8
            ids = ids[ids >= 0]
            step = 1 if hi - lo <= 32 else 32
            for k in range(0, ids.size, step):
                part = ids[k:k + step][hit[i, ids[k:k + step]]]
                if part.size:
                    want = part[np.argmin(t[i, part])] + 8
                    seen.add((step, k > 0))
                    break
            if want != shn.SHN_MISS:
                assert abs(gt[i] - t[i, want - 8]) <= 1e-6 * 2.0
                break
        assert got[i] == want
    assert len(seen) > 1


@pytest.mark.parametrize("what,tris,res,rays", [
    ("ball", 30000, (21, 21, 21), 5003),     # empty cells around cells of thousands of references
    ("ball", 30000, (90, 88, 91), 140001),   # up to ~200 references in a cell, short ranges around
    ("large", 1500, (33, 32, 31), 20011),    # triangles of many cells, missing from some that they cross
    ("large", 6000, (9, 10, 8), 4001),       # the same in long ranges
    ("plates", 4000, (40, 3, 3), 3001),      # long thin triangles across whole rows of cells
])
def test_dense_cells(gpu, what, tris, res, rays):
    """Closest and any hits, from arrays and from a camera, where cells are crowded or triangles are large
    against them: bit for bit those of the oracle."""
    import torch

    import shinobi_b200 as shn
    r = np.random.RandomState(tris + res[0])
    if what == "ball":
        c = r.normal(size=(tris, 1, 3))
        c = 0.5 + 0.04 * c / np.linalg.norm(c, axis=2, keepdims=True) * r.uniform(0, 1, (tris, 1, 1)) ** (1 / 3)
        c[::10] = r.uniform(0, 1, (len(c[::10]), 1, 3))
        v = c + r.uniform(-0.004, 0.004, (tris, 3, 3))
    elif what == "large":
        v = r.uniform(0.2, 0.8, (tris, 1, 3)) + r.uniform(-0.2, 0.2, (tris, 3, 3))
    else:
        v = r.uniform(0.0, 1.0, (tris, 1, 3)) + r.uniform(-1, 1, (tris, 3, 3)) * np.array([0.5, 0.02, 0.02])
    v = v.reshape(-1, 3).astype(np.float32)
    idx = np.arange(3 * tris, dtype=np.uint32).reshape(-1, 3)
    b = oracle.bounds(v, idx)
    og = oracle.build_uniform(v, idx, b, np.array(res, np.int32))
    g = shn.Grid().build(shn.FaceSoup(v, idx), shn.grid_params(shn.SHN_GRID_UNIFORM, res=res))
    org, d, tmax = _rays(rays, b, seed=7)
    near = np.arange(rays) % 3 != 0  # two of three rays aim at the crowd
    aim = 0.5 + r.uniform(-0.05, 0.05, (rays, 3)) - org
    aim /= np.maximum(1e-6, np.linalg.norm(aim, axis=1, keepdims=True))
    d[near] = aim[near].astype(np.float32)
    dev = [torch.from_numpy(x).cuda() for x in (org, d, tmax)]
    h = g.trace_closest(*dev)
    ref = oracle.trace_closest(og, org, d, tmax)
    for name, x, y in zip(("tri", "t", "u", "v"), (h.tri, h.t, h.u, h.v), ref):
        assert np.array_equal(x.cpu().numpy().view(np.uint32), np.ascontiguousarray(y).view(np.uint32)), name
    assert (h.tri != -1).any()
    occ = g.trace_any(*dev).cpu().numpy()
    assert np.array_equal(occ, np.asarray(oracle.trace_any(og, org, d, tmax)[0]).astype(np.uint8))
    cam = scenes.Camera((0.4, -0.7, 0.6), (0.1, 1.2, -0.1), (0.0, 0.0, 1.0), 30.0, 131, 89)
    c = g.trace_primary(cam)
    co, cd = oracle.primary_rays(cam)
    ref = oracle.trace_closest(og, co, cd)
    for name, x, y in zip(("tri", "t", "u", "v"), (c.tri, c.t, c.u, c.v), ref):
        assert np.array_equal(x.cpu().numpy().view(np.uint32), np.ascontiguousarray(y).view(np.uint32)), name


@pytest.mark.parametrize("kind", [0, 1])
def test_rays_in_negated_views(gpu, kind):
    """Rays whose memory holds the negated values (the imaginary part of a conjugate) are not read in place."""
    import torch

    import shinobi_b200 as shn
    sc = scenes.uniform_soup(5000, seed=3)
    g = shn.Grid().build(shn.FaceSoup(sc.vertices, sc.indices), shn.grid_params(kind))
    rays = [torch.from_numpy(x).cuda() for x in _rays(1003, oracle.bounds(sc.vertices, sc.indices), seed=5)]
    neg = [torch.complex(torch.zeros_like(x), -x).conj().imag for x in rays]
    assert all(x.is_neg() and torch.equal(x, y) for x, y in zip(neg, rays))
    ref, occ = g.trace_closest(*rays), g.trace_any(*rays)
    assert (ref.tri != -1).any()
    for k in ((1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)):
        r = [neg[i] if k[i] else rays[i] for i in range(3)]
        h = g.trace_closest(*r)
        assert torch.equal(h.tri, ref.tri) and torch.equal(h.t.view(torch.int32), ref.t.view(torch.int32))
        assert torch.equal(g.trace_any(*r), occ)
