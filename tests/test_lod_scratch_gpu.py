"""Joins under memory caps that leave no room for the LOD loop's queues: they
run as one warp per voxel pair and return the same; the queues of one join make
room for what is allocated after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("self_join,kw", [(False, dict(query="nn", knn=3)), (False, dict(query="within", within=150.0)),
                                          (True, dict(query="within", within=60.0))])
def test_joins_under_caps_return_the_same(pkg, ctx, self_join, kw):
    a, b = pkg.tdp.gen_tiles(10, 60, seed=91)
    T1, T2 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    q, t, d = ctx.join(T1, None if self_join else T2, form=pkg.FORM_TUNED, **kw)
    want = ctx.stats()["full_evals"]
    T1.free()
    T2.free()
    forms = set()
    for mb in range(256, 345, 4):
        with pkg.Context(0, budget_bytes=mb << 20) as small:
            try:
                S1, S2 = pkg.tdp.Tile(small, a), pkg.tdp.Tile(small, b)
                q2, t2, d2 = small.join(S1, None if self_join else S2, form=pkg.FORM_TUNED, **kw)
            except pkg.TdpError as e:
                assert not forms, (mb, e)  # a larger cap never refuses what a smaller one took
                continue
            np.testing.assert_array_equal(q2, q)
            np.testing.assert_array_equal(t2, t)
            np.testing.assert_array_equal(d2, d)
            forms.add(small.stats()["full_evals"] == want)
    assert forms == {False, True}


def test_the_queues_make_room(pkg):
    """Tiles uploaded after a join take its queues' room, down to the last that
    fits; the join then runs without them."""
    a, b = pkg.tdp.gen_tiles(10, 60, seed=91)
    _, small_b = pkg.tdp.gen_tiles(1, 60, seed=92)
    with pkg.Context(0, budget_bytes=330 << 20) as small:
        S1, S2 = pkg.tdp.Tile(small, a), pkg.tdp.Tile(small, b)
        q, t, d = small.join(S1, S2, query="nn", knn=3, form=pkg.FORM_TUNED)
        first = small.stats()["full_evals"]
        kept = []
        with pytest.raises(pkg.TdpError):
            while True:
                kept.append(pkg.tdp.Tile(small, small_b))
        kept.pop().free()
        kept.pop().free()
        q2, t2, d2 = small.join(S1, S2, query="nn", knn=3, form=pkg.FORM_TUNED)
        assert small.stats()["full_evals"] != first
    np.testing.assert_array_equal(q2, q)
    np.testing.assert_array_equal(t2, t)
    np.testing.assert_array_equal(d2, d)
