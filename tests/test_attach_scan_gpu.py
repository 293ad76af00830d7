"""The prefix arrays of an attached tile around the sizes of a block's run (4,096
voxels): the tile is read on the GPU (not handed to the host's parser by its
layout check) and joins as the uploaded tile does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv,npv,vs", [(1, 1, 100), (1, 315, 100), (4, 79, 100), (3, 210, 100), (16, 128, 320)])
def test_attached_prefixes(pkg, ctx, nv, npv, vs):
    a, b = pkg.tdp.gen_tiles(nv, npv, seed=61, voxel_size=vs)
    U, V = pkg.tdp.Tile(ctx, a), pkg.tdp.Tile(ctx, b)
    pa = pkg.tdp.pinned_copy(a)
    A = pkg.tdp.Tile(ctx, pa, attach=True)
    iu, ia = U.info(), A.info()
    assert ia["attached"] and ia["n_voxels"] == iu["n_voxels"] and list(ia["n_tris"]) == list(iu["n_tris"])
    n, nvox = ia["n_objects"], ia["n_voxels"]
    assert ia["h2d_bytes"] == n * (32 + 52) + nvox * 116  # what the GPU's pass reads
    for kw in (dict(query="within", within=150.0), dict(query="nn", knn=1)):
        want = ctx.join(U, V, form=pkg.FORM_TUNED, **kw)
        got = ctx.join(A, V, form=pkg.FORM_TUNED, **kw)
        for x, y in zip(got, want):
            np.testing.assert_array_equal(x, y)
    for t in (U, V, A):
        t.free()
