"""An autotuned context whose next join has no room for the LOD loop's queues:
that join runs with the fastest of the other configurations, not with
configuration 0's refine of one warp per voxel pair, and returns the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_without_room_the_best_other_configuration(pkg, ctx):
    a, b = pkg.tdp.gen_tiles(10, 60, seed=91)
    c, d = pkg.tdp.gen_tiles(10, 20, seed=92)
    kw = dict(query="within", within=150.0)
    T1, T2 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    ctx.set_refine_config(0)
    want = ctx.join(T1, T2, **kw)
    tasks = ctx.stats()["full_evals"]
    evals = {}
    for cfg in range(1, 18):
        ctx.set_refine_config(cfg)
        ctx.join(T1, T2, **kw)
        evals[cfg] = ctx.stats()["full_evals"]
    ctx.set_refine_config(0)
    T1.free()
    T2.free()

    def capped(mb, tune):
        with pkg.Context(0, budget_bytes=mb << 20) as small:
            if tune:
                s1, s2 = pkg.tdp.Tile(small, c), pkg.tdp.Tile(small, d)
                small.autotune(s1, s2, **kw)
                assert small.stats()["refine_items"] > 0
                s1.free()
                s2.free()
                if small.refine_config() != 0:
                    pytest.skip("the autotuner took another configuration")
            got = small.join(pkg.tdp.Tile(small, a), pkg.tdp.Tile(small, b), **kw)
            for x, y in zip(got, want):
                np.testing.assert_array_equal(x, y)
            return small.stats()["full_evals"]

    eager = None
    for mb in range(344, 255, -8):  # the largest cap without room for the queues
        n = capped(mb, False)
        if n != tasks:
            eager = n
            break
    assert eager is not None
    # per LOD the fastest of the others: its evaluations are none of eager's, and within the others' range
    n = capped(mb, True)
    assert n != eager and min(evals.values()) <= n <= max(evals.values())
