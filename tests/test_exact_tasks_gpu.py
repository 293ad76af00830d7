"""The exact-distance stage over the task kernels: against the FP64 oracle at
small and odd sizes, with more cluster pairs than its queues hold, and with and
without room for those queues under a memory cap."""
import numpy as np
import pytest

from oracle_bind import join_exact

pytestmark = pytest.mark.gpu


def _truth(a, b, self_join, query, **kw):
    q, t, d, _ = join_exact(a, None if self_join else b, self_join, query == "nn", **kw)
    return {(int(x), int(y)): float(v) for x, y, v in zip(q, t, d)}


@pytest.mark.parametrize("form", ["plain", "tuned"])
@pytest.mark.parametrize("nv,npv,vs,query,knn,tau,level,lods,self_join", [
    (1, 1, 100, "within", 0, 1000.0, 2, (20, 40, 60, 80, 100), False),
    (2, 9, 40, "within", 0, 300.0, 2, (20, 100), False),
    (2, 9, 100, "nn", 3, 0.0, 1, (60, 100), False),
    (1, 33, 300, "within", 0, 120.0, 0, (100,), True),
    (1, 20, 50, "nn", 4, 0.0, 2, (40, 80), True),
])
def test_exact_distances_equal_the_oracle(pkg, ctx, form, nv, npv, vs, query, knn, tau, level, lods, self_join):
    a, b = pkg.tdp.gen_tiles(nv, npv, seed=77, voxel_size=vs)
    T1, T2 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    truth = _truth(a, b, self_join, query, knn=max(knn, 1), tau=tau)
    q, t, d = ctx.join(T1, None if self_join else T2, query=query, knn=max(knn, 1), within=tau, lods=lods, hausdorff_level=level,
                       form=pkg.FORM_PLAIN if form == "plain" else pkg.FORM_TUNED, exact_distances=True)
    st = ctx.stats()
    T1.free()
    T2.free()
    assert len(q) > 0 and st["exact_items"] >= len(q) >= 1
    assert st["exact_dropped_items"] + st["exact_below_items"] <= st["exact_items"]
    for x, y, v in zip(q, t, d):
        if (int(x), int(y)) in truth:  # a LOD list without 100 may report other neighbours
            ref = truth[(int(x), int(y))]
            assert abs(v - ref) <= 1e-9 * max(ref, 1.0)


def test_full_queues_and_caps_give_the_same_distances(pkg, ctx):
    """Two copies of a tile: every object touches its copy everywhere, more
    cluster pairs than the queue holds.  Caps on the memory take the queues away."""
    a, _ = pkg.tdp.gen_tiles(6, 110, seed=78)
    T1, T2 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, a)
    kw = dict(query="within", within=25.0, form=pkg.FORM_TUNED, exact_distances=True)
    q, t, d = ctx.join(T1, T2, **kw)
    want = ctx.stats()["exact_full_evals"]
    T1.free()
    T2.free()
    assert (d[q == t] == 0.0).all() and (q == t).sum() == 660
    assert (d >= 0).all() and (d <= 25.0 * (1 + 1e-6)).all()
    sym = {(int(x), int(y)): v for x, y, v in zip(q, t, d)}
    for (x, y), v in sym.items():  # the distance has no direction
        assert abs(sym[(y, x)] - v) <= 1e-9 * max(v, 1.0)
    other = 0
    for mb in (450, 400, 370, 340, 320, 300, 290, 280, 270):
        with pkg.Context(0, budget_bytes=mb << 20) as small:
            try:
                S1, S2 = pkg.tdp.Tile(small, a), pkg.tdp.Tile(small, a)
                q2, t2, d2 = small.join(S1, S2, **kw)
            except pkg.TdpError:
                continue
            np.testing.assert_array_equal(q2, q)
            np.testing.assert_array_equal(t2, t)
            assert (np.abs(d2 - d) <= 1e-12 * np.maximum(d, 1.0)).all()
            other += small.stats()["exact_full_evals"] != want
    assert other > 0
