"""Bound preparation of meshes whose triangles are long and thin: their spheres
overlap everything, so that the voxels near a query decide how many FP64
distances it takes."""
import numpy as np
import pytest

from test_bounds import oracle_bounds
from test_decimate_gpu import double_cone

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,most", [(3000, 19190121), (10000, 165510334)])
def test_no_more_distances_than_all_of_each_querys_voxels(pkg, ctx, n, most):
    """most: a scan of all triangles of the voxels near each query.  Voxels near any of a warp's
    32 queries, scanned for all of them, took 28,713,699 and 278,588,640."""
    raw, _ = ctx.raw_from_meshes(*pkg.tdp.stack_meshes([double_cone(n)]), voxel_size=100)
    T = pkg.tdp.Tile(ctx, raw)
    assert 0 < ctx.compute_bounds(T)["dist_evals"] < most
    T.free()
    if n == 3000:
        np.testing.assert_array_equal(raw, oracle_bounds(raw))
