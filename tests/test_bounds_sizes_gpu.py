"""Bound preparation at the sizes where its batches of 32 queries and 64 staged
triangles can go wrong, and where distances tie: bytes equal to the FP64 oracle's."""
import numpy as np
import pytest

from rawdt import read_tile, write_tile
from test_bounds import oracle_bounds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{"voxel_size": 24, "nucleus_subdiv": 2}, {"voxel_size": 33}, {"voxel_size": 64},
                                {"voxel_size": 65}, {"voxel_size": 130}, {"voxel_size": 5000}])
def test_voxel_sizes(pkg, ctx, kw):
    nb, vb = pkg.tdp.gen_tiles(1, 3, seed=401, tube_sides=8, tube_rings=10, **kw)
    # (the generator cuts the small tube into empty voxels below 64 triangles each)
    for raw in (nb, vb) if kw["voxel_size"] >= 64 else (nb,):
        got, info = ctx.raw_compute_bounds(raw)
        np.testing.assert_array_equal(got, oracle_bounds(raw))
        assert info["facet_queries"] > 0


@pytest.mark.parametrize("shift", [0.0, 3.0e4])
def test_repeated_and_distant_triangles(pkg, ctx, shift):
    """Every triangle twice (each nearest one ties with its copy), far from the
    origin, and an object whose voxels are far apart."""
    nb, _ = pkg.tdp.gen_tiles(1, 2, seed=402)
    objs = []
    for o in read_tile(nb):
        twice = [[np.concatenate([t, t]) + np.float32(shift) for t in o.tris[li]] for li in range(5)]
        objs.append(twice)
    far = [[t + np.float32(200 * v) for v, t in enumerate(o)] for o in objs[0]]
    raw = write_tile(objs + [far])
    got, _ = ctx.raw_compute_bounds(raw)
    np.testing.assert_array_equal(got, oracle_bounds(raw))
