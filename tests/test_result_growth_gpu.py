"""Result rows as the context's page-locked buffer grows: a within join's rows
that fit come with the counters, the others after their number is known.  Each
join returns what it returns on a fresh context."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact", [False, True])
def test_joins_of_all_sizes_after_each_other(pkg, exact):
    nb, vb = pkg.tdp.gen_tiles(60, 20, seed=29, nucleus_subdiv=1)
    more = dict(exact_distances=True) if exact else {}
    joins = [dict(query="within", within=w) for w in (0.0, 90.0, 100.0, 700.0, 2500.0, 200.0, 1e5, 2500.0, 0.0)]
    joins[3:3] = [dict(query="nn", knn=2)]
    joins += [dict(query="nn", knn=59), dict(query="within", within=1500.0)]
    joins += [dict(obj_knn=np.arange(1200, dtype=np.int32) % 3, obj_within=np.full(1200, 800.0, np.float32))]
    with pkg.Context(0) as c:
        T1, T2 = pkg.tdp.Tile(c, nb), pkg.tdp.Tile(c, vb)
        got = [c.join(T1, T2, **kw, **more) for kw in joins]
    sizes = set()
    for kw, rows in zip(joins, got):
        with pkg.Context(0) as c:
            want = c.join(pkg.tdp.Tile(c, nb), pkg.tdp.Tile(c, vb), **kw, **more)
        for x, y in zip(rows, want):
            np.testing.assert_array_equal(x, y, err_msg=str(kw))
        sizes.add(len(rows[0]))
    assert 1200 * 60 in sizes and len(sizes) > 6  # above and below the rows that come at once
