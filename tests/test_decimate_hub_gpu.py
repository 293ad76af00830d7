"""Decimation around a vertex with thousands of facets: it is a third vertex of
every edge around it, and only whether it has more than three neighbours is
asked.  Tiles equal the FP64 oracle's, and a fan costs about what a sphere of as
many facets does."""
import numpy as np
import pytest

from test_bounds import oracle_bounds
from test_decimate_gpu import double_cone, grid, needle
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


def spindle(n, seed):
    """A closed tube of n rings that shrink to both ends: short edges at the ends, merged into few vertices."""
    rng = np.random.default_rng(seed)
    t = np.concatenate([-np.geomspace(50, 0.01, n // 2), np.geomspace(0.01, 50, n - n // 2)])
    a = np.arange(7) * (2 * np.pi / 7)
    V = np.concatenate([np.stack([np.full(7, z), np.cos(a), np.sin(a)], 1) * (1 + 0.01 * rng.random()) for z in t] + [[[-60, 0, 0], [60, 0, 0]]])
    F = []
    for k in range(n - 1):
        for i in range(7):
            p, q = 7 * k + i, 7 * k + (i + 1) % 7
            F += [(p, p + 7, q), (q, p + 7, q + 7)]
    for i in range(7):
        F += [(7 * n, i, (i + 1) % 7), (7 * n + 1, 7 * (n - 1) + (i + 1) % 7, 7 * (n - 1) + i)]
    return V.astype(np.float32), np.array(F, np.uint32)


@pytest.mark.parametrize("mesh", [needle(40), needle(330), spindle(300, 1), spindle(81, 2), double_cone(3000, h=300.0)])
def test_long_chains_equal_the_oracle(pkg, ctx, mesh):
    """Vertices that take in hundreds of others: their lists are rewritten without the facets that are gone."""
    meshes = [mesh, needle(12), spindle(9, 3)]
    raw, _ = ctx.raw_from_meshes(*pkg.tdp.stack_meshes(meshes), voxel_size=60)
    np.testing.assert_array_equal(raw, oracle_bounds(oracle_prep(meshes, voxel_size=60)))


def test_a_long_chain_takes_no_longer_than_a_sheet(pkg, ctx):
    """18,000 facets; 40 times as long where each round went through all that the chain had held."""
    def decimate_ms(mesh):
        m = pkg.tdp.stack_meshes([mesh])
        return min(ctx.raw_from_meshes(*m, voxel_size=100)[1]["decimate_ms"] for _ in range(3))
    assert decimate_ms(needle(1500)) < 8 * decimate_ms(grid(96, 96, 5))
