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
