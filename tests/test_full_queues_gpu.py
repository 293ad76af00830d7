"""The statistic of voxel pairs that found a queue of the LOD loop or of the
exact stage full, on the workloads that are meant to fill them, and none where
a join has few."""
import numpy as np
import pytest

from test_lod_tasks_gpu import scaled_bounds

pytestmark = pytest.mark.gpu


def test_wide_bounds(pkg, ctx):
    nb, vb = pkg.tdp.gen_tiles(3, 24, seed=305, voxel_size=5000, tube_sides=12, tube_rings=30)
    T1, T2 = pkg.tdp.Tile(ctx, scaled_bounds(nb, 40.0)), pkg.tdp.Tile(ctx, scaled_bounds(vb, 40.0))
    ctx.set_refine_config(0)
    full = []
    for kw in (dict(query="nn", knn=2), dict(query="within", within=150.0)):
        ctx.join(T1, T2, form=pkg.FORM_TUNED, **kw)
        st = ctx.stats()
        assert 0 <= st["lod_full_items"] <= st["refine_items"]
        full.append(st["lod_full_items"])
    assert max(full) > 0
    T1.free()
    T2.free()
    T1, T2 = pkg.tdp.Tile(ctx, nb), pkg.tdp.Tile(ctx, vb)
    ctx.join(T1, T2, query="nn", knn=2, form=pkg.FORM_TUNED)
    assert ctx.stats()["lod_full_items"] == 0
    T1.free()
    T2.free()


def test_objects_that_touch_everywhere(pkg, ctx):
    a, b = pkg.tdp.gen_tiles(6, 110, seed=78)
    T1, T2, T3 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    kw = dict(query="within", within=25.0, form=pkg.FORM_TUNED, exact_distances=True)
    q, t, d = ctx.join(T1, T2, **kw)
    st = ctx.stats()
    assert 0 < st["exact_full_items"] <= st["exact_items"]
    assert (d[q == t] == 0.0).all()
    ctx.join(T1, T3, **kw)
    assert ctx.stats()["exact_full_items"] == 0
    for x in (T1, T2, T3):
        x.free()


@pytest.mark.parametrize("vs", [200, 500])
@pytest.mark.parametrize("kw", [dict(query="nn", knn=5), dict(query="within", within=200.0)])
def test_larger_voxels_have_room_in_the_exact_stage(pkg, ctx, vs, kw):
    """Every candidate had room for 16 cluster pairs and 8 triangle pairs whatever its voxels' sizes:
    97,029 of 329,923 candidates of 200 triangles a voxel did not fit and were gone through by one warp each."""
    from oracle_bind import join_exact
    a, b = pkg.tdp.gen_tiles(50, 40, seed=9, voxel_size=vs)
    T1, T2 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    ctx.join(T1, T2, exact_distances=True, **kw)
    st = ctx.stats()
    assert st["exact_items"] > 20000 and st["exact_full_items"] * 100 <= st["exact_items"]
    T1.free()
    T2.free()
    a, b = pkg.tdp.gen_tiles(6, 12, seed=9, voxel_size=vs)
    T1, T2 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    q, t, d = ctx.join(T1, T2, exact_distances=True, **kw)
    tq, tt, td, _ = join_exact(a, b, False, kw["query"] == "nn", knn=kw.get("knn", 1), tau=kw.get("within", 0.0))
    truth = {(int(x), int(y)): float(v) for x, y, v in zip(tq, tt, td)}
    for x, y, v in zip(q, t, d):
        ref = truth[(int(x), int(y))]
        assert abs(v - ref) <= 1e-9 * max(ref, 1.0)
    T1.free()
    T2.free()
