"""Tiles with a triangle that is not finite: a bound that is not a number lets a
triangle pair pass, and what passes has to exist.  The bad object's own pairs
have no defined distance; every other pair's rows equal those of the
one-warp-per-voxel-pair refine (configuration 17) on the same tiles, and those
of the tiles without the bad triangle."""
import numpy as np
import pytest

from test_lod_tasks_gpu import records

pytestmark = pytest.mark.gpu


def spoiled(raw, obj, value, which):
    """Triangle `which` (0 first, -1 last) of the last voxel of object obj gets `value` at every LOD."""
    import struct
    out = raw.copy()
    mine = [r for r in records(raw) if r[0] == obj]
    _, _, at, data = mine[-1]
    sizes = []
    for li in range(5):
        off, n = struct.unpack_from("<QQ", raw, at + 16 * li)
        sizes.append(n)
        if n:
            t = data + off + 36 * (which % n)
            out[t:t + 36].view(np.float32)[4] = value
    assert any(n % 8 for n in sizes)  # a cluster with missing triangles beside it
    return out


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("which", [0, -1])
def test_other_pairs_are_untouched(pkg, value, which):
    nb, vb = pkg.tdp.gen_tiles(6, 20, seed=71, voxel_size=37)
    nq, nt = 120, 6
    with pkg.Context(0) as c:
        good1, good2 = pkg.tdp.Tile(c, nb), pkg.tdp.Tile(c, vb)
        bad1 = pkg.tdp.Tile(c, spoiled(nb, nq - 1, value, which))
        bad2 = pkg.tdp.Tile(c, spoiled(vb, nt - 1, value, which))
        cases = [(bad1, good2, kw) for kw in (dict(query="nn", knn=2), dict(query="within", within=300.0))]
        cases += [(good1, bad2, dict(query="within", within=300.0)), (bad1, None, dict(query="within", within=60.0))]
        for t1, t2, kw in cases:
            for more in (dict(), dict(hausdorff_level=1), dict(lods=[100]), dict(exact_distances=True)):
                rows = []
                for cfg, a, b in ((0, t1, t2), (17, t1, t2), (0, good1, None if t2 is None else good2)):
                    c.set_refine_config(cfg)
                    q, t, d = c.join(a, b, **kw, **more)
                    ok = (q != nq - 1) if t1 is bad1 else (t != nt - 1)
                    if t2 is None:
                        ok &= t != nq - 1
                    rows.append((q[ok], t[ok], d[ok]))
                assert len(rows[0][0])
                for other in rows[1:]:
                    for x, y in zip(rows[0], other):
                        np.testing.assert_array_equal(x, y, err_msg=f"{kw} {more}")
