"""LOD preparation under the smallest memory caps that it took before the
decimation kept lists of every vertex's facets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which,nv,npv,cap", [("nuclei", 1, 1, 438272), ("nuclei", 2, 20, 16932864), ("vessels", 1, 1, 7507968),
                                              ("vessels", 2, 1, 12443648)])
def test_smallest_caps(pkg, ctx, which, nv, npv, cap):
    m = pkg.tdp.gen_meshes(nv, npv, seed=4, which=which)
    want, _ = ctx.raw_from_meshes(*m, voxel_size=100)
    with pkg.Context(0, budget_bytes=cap) as small:
        got, _ = small.raw_from_meshes(*m, voxel_size=100)
    np.testing.assert_array_equal(got, want)
