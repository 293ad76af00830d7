"""The voxel filter at the sizes where its pruning can go wrong: objects of one
voxel, around the limits of its small form (24 tile-2 voxels), of a warp (32)
and of a chunk (64), more than 64 tile-1 voxels; early reports of a within
join.  The plain form takes the reference's own decisions, so its sets pin the
filter's ranges through every later step; the early reports' distance bounds are
restated from the voxel records, chunk by chunk."""
import numpy as np
import pytest

from rawdt import read_tile, write_tile

pytestmark = pytest.mark.gpu


def cloud(rng, n_obj, n_vox, spread):
    """Objects of n_vox voxels of one small triangle each, the same at every LOD."""
    objs = []
    for _ in range(n_obj):
        at = rng.uniform(0, spread, 3)
        tris = [(at + rng.normal(size=3) * 8 + rng.normal(size=(3, 3))).astype(np.float32).reshape(1, 9) for _ in range(n_vox)]
        objs.append([tris] * 5)
    return write_tile(objs)


def ranges(A, B, tau, chunk=64):
    """(nearest box gap, nearest core distance or the one an early report stops at) of two objects."""
    lo1, hi1, c1 = (A[:, None, 3 * k:3 * k + 3].astype(np.float64) for k in range(3))
    lo2, hi2, c2 = (B[None, :, 3 * k:3 * k + 3].astype(np.float64) for k in range(3))
    gap = np.sqrt((np.maximum(np.maximum(lo1 - hi2, lo2 - hi1), 0) ** 2).sum(-1))
    core = np.sqrt(((c1 - c2) ** 2).sum(-1))
    if len(B) >= 24:
        for a in range(0, len(A), chunk):
            for b in range(0, len(B), chunk):
                seen = core[:a + chunk].min() if b + chunk >= len(B) else min(
                    core[:a].min() if a else np.inf, core[a:a + chunk, :b + chunk].min())
                if seen * (1 + 1e-6) <= tau:
                    return gap.min(), seen, True
    return gap.min(), core.min(), False


@pytest.mark.parametrize("n1,n2", [(1, 1), (1, 200), (13, 23), (13, 24), (32, 33), (33, 64), (65, 65), (130, 129)])
def test_early_reports_and_sets(pkg, ctx, n1, n2):
    rng = np.random.default_rng(n1 * 1000 + n2)
    nb, vb = cloud(rng, 40, n1, 120.0), cloud(rng, 25, n2, 120.0)
    N, V = read_tile(nb), read_tile(vb)
    T1, T2 = pkg.tdp.Tile(ctx, nb), pkg.tdp.Tile(ctx, vb)
    tau = 60.0
    q, t, d = ctx.join(T1, T2, query="within", within=tau)
    got = {(a, b): x for a, b, x in zip(q.tolist(), t.tolist(), d.tolist())}
    for i in range(len(N)):
        for j in range(len(V)):
            mn, mx, early = ranges(N[i].voxels, V[j].voxels, tau)
            if mx <= tau * (1 - 1e-5):
                # decided by the filter: reported with its core distance
                assert abs(got[(i, j)] - mx) <= 1e-5 * (mx + 1), (i, j, early)
            elif mn > tau * (1 + 1e-5):
                assert (i, j) not in got
    for args in (dict(query="within", within=tau), dict(query="intersect")):
        want = ctx.join(T1, T2, form=pkg.FORM_PLAIN, **args)
        have = ctx.join(T1, T2, form=pkg.FORM_TUNED, **args)
        for k in range(2):
            np.testing.assert_array_equal(have[k], want[k])
    T1.free()
    T2.free()
