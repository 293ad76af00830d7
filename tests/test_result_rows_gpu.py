"""Rows of a join where they take another way back: copied with the counters or,
above 16 MB, after their number was read; ordered by a warp per query, with each block adding up the
counts before it (up to 4,096 queries) or a scan, or by the general sort (kNN
with more than 512 candidates of a query)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ordered(q, t):
    k = q.astype(np.int64) << 32 | t
    assert (np.diff(k) > 0).all()
    return k


@pytest.mark.parametrize("nv,npv,kw", [
    (3, 40, dict(query="within", within=0.0)),                      # few or no rows
    (8, 512, dict(query="nn", knn=1)),                              # 4,096 queries
    (17, 241, dict(query="nn", knn=1)),                             # 4,097
    (17, 241, dict(query="within", within=250.0)),
    (17, 241, dict(query="nn", knn=5)),
])
def test_rows_equal_those_of_shards(pkg, ctx, nv, npv, kw):
    a, b = pkg.tdp.gen_tiles(nv, npv, seed=17, nucleus_subdiv=1)
    T1, T2 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    q, t, d = ctx.join(T1, T2, form=pkg.FORM_TUNED, **kw)
    ordered(q, t)
    n, got = nv * npv, []
    for lo, hi in ((0, 1), (1, n // 5), (n // 5, n - 1), (n - 1, n)):
        got.append(ctx.join(T1, T2, form=pkg.FORM_TUNED, query_range=(lo, hi), **kw))
    for k, x in enumerate((q, t, d)):
        np.testing.assert_array_equal(np.concatenate([g[k] for g in got]), x)
    if kw["query"] == "nn":
        np.testing.assert_array_equal(q, np.repeat(np.arange(n), kw["knn"]))
    T1.free()
    T2.free()


@pytest.mark.parametrize("knn", [511, 512, 513, 700])
def test_many_neighbours_are_the_candidates(pkg, ctx, knn):
    """Every object is a result when K is all there are: ids in order, both forms."""
    a, _ = pkg.tdp.gen_tiles(3, 234, seed=18, nucleus_subdiv=1)
    T = pkg.tdp.Tile(ctx, a)
    q, t, d = ctx.join(T, None, query="nn", knn=knn, form=pkg.FORM_TUNED)
    ordered(q, t)
    assert len(q) == 702 * min(knn, 701) and (q != t).all()
    T.free()


def test_more_rows_than_come_back_at_once(pkg, ctx):
    a, _ = pkg.tdp.gen_tiles(12, 100, seed=19, nucleus_subdiv=1)
    T = pkg.tdp.Tile(ctx, a)
    for kw in (dict(), dict(exact_distances=True)):
        q, t, d = ctx.join(T, None, query="within", within=1e5, form=pkg.FORM_TUNED, **kw)
        ordered(q, t)
        assert len(q) == 1200 * 1199 and len(d) == len(q) and (d >= 0).all()
    T.free()


def test_mixed_queries(pkg, ctx):
    a, b = pkg.tdp.gen_tiles(10, 30, seed=20, nucleus_subdiv=1)
    T1, T2 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    rng = np.random.default_rng(3)
    knn = rng.integers(0, 4, 300).astype(np.int32)
    tau = np.where(knn == 0, 200.0, 0.0).astype(np.float32)
    q, t, d = ctx.join(T1, T2, obj_knn=knn, obj_within=tau, form=pkg.FORM_TUNED)
    ordered(q, t)
    wq, wt, _ = ctx.join(T1, T2, query="within", within=200.0, form=pkg.FORM_TUNED)
    for i in range(300):
        if knn[i]:
            kq, kt, _ = ctx.join(T1, T2, query="nn", knn=int(knn[i]), query_range=(i, i + 1), form=pkg.FORM_TUNED)
            np.testing.assert_array_equal(t[q == i], kt)
        else:
            np.testing.assert_array_equal(t[q == i], wt[wq == i])
    T1.free()
    T2.free()
