"""New vertices under a built grid: until the next build, every trace answers for the triangles that the
grid was built from, and for the new ones after it."""
import numpy as np
import pytest

import oracle
from shinobi_b200 import scenes

pytestmark = pytest.mark.gpu


def _update(shn, soup, how, new):
    import torch
    if how == "host":
        soup.update_vertices(new)
    elif how == "device":
        soup.update_vertices(torch.from_numpy(new).cuda())
    elif how == "interpolate":
        k = torch.from_numpy(new).cuda()
        soup.interpolate_vertices(k, k, 0.0)
    else:  # refused, after it has overwritten the scene's vertices
        with pytest.raises(shn.ShinobiError):
            soup.update_vertices(torch.full(new.shape, float("nan"), device="cuda"))


@pytest.mark.parametrize("how", ["host", "device", "interpolate", "refused"])
@pytest.mark.parametrize("tris,kind,sat", [(1, 0, 0), (33, 0, 0), (5000, 0, 0), (5000, 0, 1), (5000, 1, 0)])
def test_vertices_updated_under_a_grid(gpu, tris, kind, sat, how):
    import torch

    import shinobi_b200 as shn
    sc = scenes.uniform_soup(tris, seed=tris, offset_scale=0.04 if tris > 100 else 0.3)
    new = np.ascontiguousarray(sc.vertices[::-1] * 0.5 + np.float32(0.25))
    soup = shn.FaceSoup(sc.vertices, sc.indices)
    p = shn.grid_params(kind, insertion=shn.SHN_INSERT_SAT if sat else shn.SHN_INSERT_PLANE)
    g = shn.Grid().build(soup, p)
    r = np.random.RandomState(3)
    n = 4001
    org = r.uniform(-0.5, 1.5, (n, 3)).astype(np.float32)
    d = r.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    tmax = np.full(n, 5.0, np.float32)
    rays = [torch.from_numpy(x).cuda() for x in (org, d, tmax)]
    cam = scenes.Camera((-1.0, -0.8, 1.4), (1.4, 1.2, -0.8), (0.0, 0.0, 1.0), 45.0, 61, 47)

    def traced():
        out = []
        cnt = torch.zeros(2, dtype=torch.int64, device="cuda")
        for stats in (None, cnt):  # the counting kernels are another engine
            shn.default_context().lib.shn_grid_set_stats(g.handle, None if stats is None else shn._ptr(stats))
            h, c = g.trace_closest(*rays), g.trace_primary(cam)
            out += [h.tri, h.t, c.tri, c.t, g.trace_any(*rays)]
        shn.default_context().lib.shn_grid_set_stats(g.handle, None)
        return [x.cpu().numpy() for x in out]

    def oracle_says(v):
        b = oracle.bounds(v, sc.indices)
        og = oracle.build_uniform(v, sc.indices, b, oracle.resolution(tris, b, 5.0))
        return og, oracle.trace_closest(og, org, d, tmax)

    before = traced()
    if kind == 0 and not sat:
        og, ref = oracle_says(sc.vertices)
        assert np.array_equal(before[0].view(np.uint32), ref[0])
    assert (before[0] != -1).any()
    _update(shn, soup, how, new)
    for a, b in zip(traced(), before):
        assert np.array_equal(a, b)
    if how == "refused":
        return
    g.build(soup, p)
    after = traced()
    assert not np.array_equal(after[0], before[0])
    if kind == 0 and not sat:
        og, ref = oracle_says(new)
        assert np.array_equal(after[0].view(np.uint32), ref[0])
        assert np.array_equal(after[1].view(np.uint32), ref[1].view(np.uint32))
