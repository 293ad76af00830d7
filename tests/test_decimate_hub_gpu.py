"""Decimation around a vertex with thousands of facets: it is a third vertex of
every edge around it, and only whether it has more than three neighbours is
asked.  Tiles equal the FP64 oracle's, and a fan costs about what a sphere of as
many facets does."""
import numpy as np
import pytest

from test_bounds import oracle_bounds
from test_decimate_gpu import double_cone, grid
from test_lodprep import oracle_prep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 6, 31, 64, 1500])
def test_fans_equal_the_oracle(pkg, ctx, n):
    meshes = [double_cone(n), double_cone(n, h=0.01)]
    raw, _ = ctx.raw_from_meshes(*pkg.tdp.stack_meshes(meshes), voxel_size=50)
    np.testing.assert_array_equal(raw, oracle_bounds(oracle_prep(meshes, voxel_size=50)))


def test_a_fan_takes_no_longer_than_a_sheet(pkg, ctx):
    """20,000 facets each; 27 times as long where each round went round both apexes."""
    def decimate_ms(mesh):
        m = pkg.tdp.stack_meshes([mesh])
        return min(ctx.raw_from_meshes(*m, voxel_size=100)[1]["decimate_ms"] for _ in range(3))
    assert decimate_ms(double_cone(10000)) < 8 * decimate_ms(grid(101, 101, 5))
