"""Joins under the smallest memory caps that they took when no scratch was
optional: queues, prefetch lists and refine parts give way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXACT = dict(query="within", within=200.0, exact_distances=True)
# (uploaded, attached) smallest caps in steps of 64 KB, of the 600 x 10 workload
CAPS = [(dict(query="nn", knn=5), 274989056, 146931712), (dict(query="within", within=300.0), 273678336, 145620992),
        (EXACT, 280100864, 151977984), (dict(query="nn", knn=3, exact_distances=True), 295305216, 167182336)]


@pytest.mark.parametrize("kw,uploaded,attached", CAPS)
def test_smallest_caps(pkg, ctx, kw, uploaded, attached):
    a, b = pkg.tdp.gen_tiles(10, 60, seed=91)
    T1, T2 = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    want = ctx.join(T1, T2, **kw)
    T1.free()
    T2.free()
    pa, pb = pkg.tdp.pinned_copy(a), pkg.tdp.pinned_copy(b)
    for cap, x, y, attach in ((uploaded, a, b, False), (attached, pa, pb, True)):
        with pkg.Context(0, budget_bytes=cap) as small:
            got = small.join(pkg.tdp.Tile(small, x, attach=attach), pkg.tdp.Tile(small, y, attach=attach), **kw)
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g, w)


def test_a_larger_attached_exact_join(pkg):
    a, b = pkg.tdp.gen_tiles(30, 100, seed=92, voxel_size=60)
    pa, pb = pkg.tdp.pinned_copy(a), pkg.tdp.pinned_copy(b)
    with pkg.Context(0, budget_bytes=705560576) as small:
        small.join(pkg.tdp.Tile(small, pa, attach=True), pkg.tdp.Tile(small, pb, attach=True), **EXACT)


def test_refine_parts_make_room(pkg):
    """A tile that fits beside what a refine batch needs at the least fits after a batch that was cut into parts."""
    rng = np.random.default_rng(5)
    n = rng.integers(1, 131, (300, 2))
    cnt = n.reshape(-1)
    end = np.cumsum(cnt)
    start = end - cnt
    tri = rng.normal(size=(int(end[-1]), 9)).astype(np.float32)
    hd = np.abs(rng.normal(size=(int(end[-1]), 2))).astype(np.float32)
    rows = np.stack([start[0::2], n[:, 0], start[1::2], n[:, 1]], 1).astype(np.uint64)
    _, b = pkg.tdp.gen_tiles(1, 1, seed=92)

    def takes(cap, form):
        with pkg.Context(0, budget_bytes=cap) as small:
            try:
                small.refine_batch(tri, hd, rows, form=form)
                pkg.tdp.Tile(small, b)
            except pkg.TdpError:
                return False
        return True

    lo, hi = 1, 1 << 16  # the plain form has no parts
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if takes(mid << 12, pkg.FORM_PLAIN) else (mid, hi)
    assert takes(hi << 12, pkg.FORM_TUNED)
