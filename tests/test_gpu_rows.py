"""Key emission from the rows kept by the count: groups whose rows fit, groups
whose rows do not (large triangles exceed the room of a first build), both in
one build, one-item and ragged last groups.  Grids must equal the oracle's, on
a first build and on the next ones, whose buffers have grown; under a memory
budget a first build keeps no rows."""
import numpy as np
import pytest

import oracle
from shinobi_b200 import scenes

pytestmark = pytest.mark.gpu


def _mixed(n, small, large, every):
    """A soup whose every `every`-th triangle is large."""
    a = scenes.uniform_soup(n, seed=n, offset_scale=small)
    b = scenes.uniform_soup(n, seed=n + 1, offset_scale=large)
    v = a.vertices.reshape(n, 9).copy()
    v[::every] = b.vertices.reshape(n, 9)[::every]
    return v.reshape(3 * n, 3), a.indices


@pytest.mark.parametrize("n,small,large,every,res", [
    (1, 0.3, 0.3, 1, (64, 3, 5)),
    (33, 0.4, 0.4, 1, (40, 41, 39)),       # no group fits
    (1000, 0.002, 0.4, 400, (30, 30, 30)),  # some do not
    (5000, 0.01, 0.02, 2, (50, 51, 52)),    # all fit
    (70, 0.5, 0.5, 1, (2048, 2, 2)),        # the longest rows
])
@pytest.mark.parametrize("kind,budget", [(0, False), (1, False), (0, True), (1, True)])
def test_kept_rows(gpu, n, small, large, every, res, kind, budget):
    import shinobi_b200 as shn
    v, i = _mixed(n, small, large, every)
    b = oracle.bounds(v, i)
    if kind == 0:
        p = shn.grid_params(shn.SHN_GRID_UNIFORM, res=res)
        og = oracle.build_uniform(v, i, b, np.array(res, np.int32))
    else:
        res = tuple(max(2, r // 8) for r in res)
        p = shn.grid_params(shn.SHN_GRID_TWO_LEVEL, lambda_leaf=4.0, leaf_threshold=2, res=res)
        og = oracle.build_two_level(v, i, b, np.array(res, np.int32), 4.0, 2)
    ctx = shn.Context(0, 8 << 30) if budget else gpu
    soup = shn.FaceSoup(v, i, ctx=ctx)
    g = shn.Grid(ctx=ctx)
    for _ in range(3):
        g.build(soup, p)
        ex = g.export()
        for k in ("cells", "indices", "top_pairs") + (("leaves",) if kind else ()):
            assert np.array_equal(ex[k], getattr(og, k)), k
