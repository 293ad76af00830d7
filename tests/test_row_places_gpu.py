"""Places of a join's rows in the block of the last query (8 queries a block),
where one warp also publishes the number of rows: every size of that block, and
the sizes around 4,096 queries where the places come from a scan instead."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def workload(pkg, ctx):
    nb, vb = pkg.tdp.gen_tiles(9, 456, seed=23, nucleus_subdiv=1)  # 4,104 nuclei
    T2 = pkg.tdp.Tile(ctx, vb)
    yield nb, pkg.tdp.raw_object_offsets(nb), T2
    T2.free()


def equal_to_shards(pkg, ctx, nb, off, T2, n, cuts, kw):
    T1 = pkg.tdp.Tile(ctx, pkg.tdp.raw_slice(nb, off, 0, n))
    shards = [ctx.join(T1, T2, form=pkg.FORM_TUNED, query_range=r, **kw) for r in zip(cuts, cuts[1:])]
    for _ in range(3):
        q, t, d = ctx.join(T1, T2, form=pkg.FORM_TUNED, **kw)
        for k, x in enumerate((q, t, d)):
            np.testing.assert_array_equal(np.concatenate([s[k] for s in shards]), x, err_msg=f"{n} {kw}")
        if kw["query"] == "nn":
            np.testing.assert_array_equal(q, np.repeat(np.arange(n), kw["knn"]))
    T1.free()


QUERIES = [dict(query="nn", knn=1), dict(query="nn", knn=7), dict(query="within", within=300.0)]


@pytest.mark.parametrize("kw", QUERIES)
def test_up_to_three_blocks(pkg, ctx, workload, kw):
    for n in range(1, 18):
        equal_to_shards(pkg, ctx, *workload, n, list(range(n + 1)), kw)


@pytest.mark.parametrize("kw", QUERIES)
@pytest.mark.parametrize("n", range(4089, 4098))
def test_around_the_scan(pkg, ctx, workload, n, kw):
    equal_to_shards(pkg, ctx, *workload, n, [0, 1, 2048, 4085, n - 2, n - 1, n], kw)
