"""Candidates on the GPU around the sizes where their order comes from another
kernel (512 candidates of a query), ring searches that end at every ring or see
fewer than K points, and transforms that coincide (ties by id): the same lists
as the host grid's."""
import numpy as np
import pytest

from rawdt import read_tile

pytestmark = pytest.mark.gpu


def _boxes(raw):
    objs = read_tile(raw)
    return np.stack([o.box for o in objs]), np.stack([o.transform for o in objs])


@pytest.fixture(scope="module")
def tiles(pkg, ctx):
    raws = [pkg.tdp.gen_tiles(1, 33, seed=51)[0], pkg.tdp.gen_tiles(6, 100, seed=52)[0]]
    T = [pkg.tdp.Tile(ctx, r) for r in raws]
    yield T, [_boxes(r) for r in raws]
    for t in T:
        t.free()


@pytest.mark.parametrize("self_join", [False, True])
@pytest.mark.parametrize("knn", [1, 2, 31, 32, 33, 100, 510, 511, 512, 513, 599, 600, 601])
def test_knn_lists_equal_the_host_grids(pkg, ctx, tiles, knn, self_join):
    T, B = tiles
    a = 1 if self_join else 0
    off, ids = pkg.tdp.tile_candidates(ctx, T[a], None if self_join else T[1], knn=knn)
    hoff, hids = pkg.tdp.candidates(*B[a], *B[1], self_join=self_join, knn=knn)
    np.testing.assert_array_equal(off, hoff)
    np.testing.assert_array_equal(ids, hids)


def test_within_lists_equal_the_host_grids_past_512(pkg, ctx, tiles):
    T, B = tiles
    seen = set()
    for tau in (0.0, 20.0, 200.0, 500.0, 600.0, 650.0, 700.0, 2000.0):
        off, ids = pkg.tdp.tile_candidates(ctx, T[0], T[1], within=tau)
        hoff, hids = pkg.tdp.candidates(*B[0], *B[1], within=tau)
        np.testing.assert_array_equal(off, hoff)
        np.testing.assert_array_equal(ids, hids)
        seen.add(int(np.diff(off).max()) > 512)
    assert seen == {False, True}


def test_coinciding_transforms_are_ordered_by_id(pkg, ctx):
    raw, _ = pkg.tdp.gen_tiles(1, 40, seed=53)
    raw = np.concatenate([raw] + [raw[1:]] * 3)  # every object four times
    T = pkg.tdp.Tile(ctx, raw)
    b, x = _boxes(raw)
    for knn in (1, 3, 4, 5, 8):
        for s in (False, True):
            off, ids = pkg.tdp.tile_candidates(ctx, T, None if s else T, knn=knn)
            hoff, hids = pkg.tdp.candidates(b, x, b, x, self_join=True, knn=knn)
            np.testing.assert_array_equal(off, hoff)
            np.testing.assert_array_equal(ids, hids)
    T.free()


@pytest.mark.parametrize("nv,npv", [(1, 1), (5, 205), (16, 1024), (5, 3277)])
def test_offsets_where_the_scan_changes(pkg, ctx, nv, npv):
    """1, 1,025, 16,384 and 16,385 queries: one block's scan, or the general one."""
    raw, _ = pkg.tdp.gen_tiles(nv, npv, seed=54, nucleus_subdiv=1, only="nuclei")
    T = pkg.tdp.Tile(ctx, raw)
    b, x = _boxes(raw)
    off, ids = pkg.tdp.tile_candidates(ctx, T, None, within=3.0)
    hoff, hids = pkg.tdp.candidates(b, x, b, x, self_join=True, within=3.0)
    np.testing.assert_array_equal(off, hoff)
    np.testing.assert_array_equal(ids, hids)
    T.free()
