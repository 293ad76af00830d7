"""The LOD loop as task kernels (refine configuration 0, csrc/lod_kernels.cu)
where it can go wrong: voxels that are empty at a later LOD (their pairs keep a
cap per voxel pair), bounds that do not hold (the last LOD is done again
without the caps), voxels of one to a few thousand triangles (cluster
remainders, queues that run full), LOD lists of every kind.  Each join must
return exactly what the one-warp-per-voxel-pair refine (configuration 17)
returns, ids and distance bounds, and the FP64 exact set where the bounds hold.
"""
import struct

import numpy as np
import pytest

from join_cases import exact_truth

pytestmark = pytest.mark.gpu


def records(raw):
    """(object, voxel, position of its 5 (offset, count) words, data start) of RAW tile bytes."""
    pos, o = 1, 0
    while pos < len(raw):
        (ds,) = struct.unpack_from("<Q", raw, pos)
        data = pos + 8
        (vn,) = struct.unpack_from("<Q", raw, data + ds)
        p = data + ds + 8 + 40
        for v in range(vn):
            yield o, v, p + 36, data
            p += 116
        pos = p + 12
        o += 1


def emptied(raw, lods, every):
    """Every `every`-th voxel loses its triangles at the given LOD indices."""
    out = raw.copy()
    for k, (_, _, at, _) in enumerate(records(raw)):
        if k % every == 0:
            for li in lods:
                struct.pack_into("<Q", out, at + 16 * li + 8, 0)
    return out


def scaled_bounds(raw, f):
    """Every triangle's (proxy, hausdorff) times f: below 1 they no longer hold."""
    out = raw.copy()
    for _, _, at, data in records(raw):
        for li in range(5):
            off, n = struct.unpack_from("<QQ", raw, at + 16 * li)
            b = data + off + 36 * n
            out[b:b + 8 * n].view(np.float32)[:] *= np.float32(f)
    return out


def joins(nq):
    return [(False, dict(query="nn", knn=2)), (False, dict(query="within", within=150.0)),
            (True, dict(query="nn", knn=min(4, nq - 1))), (True, dict(query="within", within=60.0)),
            (True, dict(query="within", within=0.0)), (True, dict(query="intersect"))]


def check(pkg, nb, vb, lods=(None,), levels=(2,), truth=False):
    with pkg.Context(0) as c:
        T1, T2 = pkg.tdp.Tile(c, nb), pkg.tdp.Tile(c, vb)
        nq = T1.info()["n_objects"]
        looped = 0
        for own, args in joins(nq):
            for ls in lods:
                for level in levels:
                    got = {}
                    for cfg in (0, 17):
                        c.set_refine_config(cfg)
                        got[cfg] = c.join(T1, None if own else T2, lods=ls, hausdorff_level=level, **args)
                        looped += c.stats()["refine_items"] > 0
                    for a, b in zip(got[0], got[17]):
                        np.testing.assert_array_equal(a, b, err_msg=f"{args} {ls} level {level}")
                    if truth and ls is None and level == 2 and args["query"] != "intersect":
                        want, margin = exact_truth(nb, vb, own, args["query"], args.get("knn", 0), args.get("within", 0.0))
                        if margin >= 1e-3:
                            assert set(zip(got[0][0].tolist(), got[0][1].tolist())) == want
        assert looped  # some of the joins refine
        T1.free()
        T2.free()


LISTS = (None, [100], [20, 100], [20, 40], [60])


@pytest.mark.parametrize("kw", [{}, {"voxel_size": 30}, {"nucleus_subdiv": 1, "voxel_size": 20},
                                {"nucleus_subdiv": 2, "voxel_size": 1 << 20}])
def test_lists_levels_and_voxel_sizes(pkg, kw):
    nb, vb = pkg.tdp.gen_tiles(5, 14, seed=301, **kw)
    check(pkg, nb, vb, lods=LISTS, levels=(0, 1, 2), truth=True)


@pytest.mark.parametrize("lods,every", [((1,), 3), ((2, 3), 2), ((1, 2, 3), 1), ((4,), 5)])
def test_voxels_empty_at_later_lods(pkg, lods, every):
    nb, vb = pkg.tdp.gen_tiles(4, 16, seed=302, voxel_size=60)
    check(pkg, emptied(nb, lods, every), emptied(vb, lods, every + 1), lods=LISTS, levels=(0, 1, 2))


@pytest.mark.parametrize("f", [0.0, 0.3, 0.9])
def test_bounds_that_do_not_hold(pkg, f):
    nb, vb = pkg.tdp.gen_tiles(4, 20, seed=303)
    check(pkg, scaled_bounds(nb, f), scaled_bounds(vb, f), lods=(None, [20, 100], [40, 60]), levels=(2,))


def test_bounds_that_do_not_hold_and_empty_voxels(pkg):
    nb, vb = pkg.tdp.gen_tiles(4, 20, seed=304, voxel_size=80)
    check(pkg, emptied(scaled_bounds(nb, 0.2), (2,), 3), emptied(scaled_bounds(vb, 0.2), (2,), 4), lods=(None, [20, 60, 100]))


def test_wide_bounds_fill_the_queues(pkg):
    """Bounds wide enough that nearly every triangle pair can matter: more
    cluster and triangle pairs than the queues hold."""
    nb, vb = pkg.tdp.gen_tiles(3, 24, seed=305, voxel_size=5000, tube_sides=12, tube_rings=30)
    check(pkg, scaled_bounds(nb, 40.0), scaled_bounds(vb, 40.0), lods=(None, [80, 100]))
