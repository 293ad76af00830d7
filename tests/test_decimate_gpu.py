"""Decimation where its vertex lists and merge chains can go wrong: a vertex with
hundreds of facets (several rows of a warp, more touched groups than the round's
list holds), a vertex at the end of a long chain, strips and bow-ties, the limits
of the storage forms.  Tiles equal, byte for byte, the FP64 oracle's."""
import numpy as np
import pytest

from test_bounds import oracle_bounds
from test_lodprep import oracle_prep

pytestmark = pytest.mark.gpu


def double_cone(n, r=10.0, h=4.0):
    """n facets around each of two apexes: vertices of degree n."""
    a = np.arange(n) * (2 * np.pi / n)
    rim = np.stack([r * np.cos(a), r * np.sin(a) * 1.1, 0.1 * np.sin(5 * a)], 1)
    V = np.concatenate([rim, [[0.3, 0.1, h], [0.0, -0.2, -h]]])
    i = np.arange(n)
    j = (i + 1) % n
    F = np.concatenate([np.stack([i, j, np.full(n, n)], 1), np.stack([j, i, np.full(n, n + 1)], 1)])
    return V.astype(np.float32), F.astype(np.uint32)


def grid(nx, ny, seed):
    """An open, bumpy sheet."""
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    V = np.stack([x, y, 0.3 * rng.normal(size=x.shape)], -1).reshape(-1, 3)
    q = (np.arange(nx - 1)[:, None] * ny + np.arange(ny - 1)[None]).reshape(-1)
    F = np.concatenate([np.stack([q, q + ny, q + 1], 1), np.stack([q + 1, q + ny, q + ny + 1], 1)])
    return V.astype(np.float32), F.astype(np.uint32)


def needle(n):
    """A closed tube whose short edges all sit at one end: collapses chain up."""
    t = np.linspace(0, 1, n) ** 3 * 50
    a = np.arange(6) * (np.pi / 3)
    V = np.concatenate([np.stack([np.full(6, z), np.cos(a) * (1 + 0.01 * z), np.sin(a)], 1) for z in t] + [[[-0.1, 0, 0], [50.5, 0, 0]]])
    F = []
    for k in range(n - 1):
        for i in range(6):
            p, q = 6 * k + i, 6 * k + (i + 1) % 6
            F += [(p, p + 6, q), (q, p + 6, q + 6)]
    for i in range(6):
        F += [(6 * n, i, (i + 1) % 6), (6 * n + 1, 6 * (n - 1) + (i + 1) % 6, 6 * (n - 1) + i)]
    return V.astype(np.float32), np.array(F, np.uint32)


@pytest.mark.parametrize("name,mesh", [("cone33", double_cone(33)), ("cone700", double_cone(700)), ("sheet", grid(23, 31, 1)),
                                       ("sheet_large", grid(90, 95, 2)), ("needle", needle(160)), ("fan4", double_cone(4))])
def test_meshes_equal_the_oracle(pkg, ctx, name, mesh):
    meshes = [mesh, needle(5), mesh]
    V, vo, F, fo = pkg.tdp.stack_meshes(meshes)
    raw, info = ctx.raw_from_meshes(V, vo, F, fo, voxel_size=40)
    want = oracle_bounds(oracle_prep(meshes, voxel_size=40))
    np.testing.assert_array_equal(raw, want)
    assert info["n_objects"] == 3


@pytest.mark.parametrize("mb", [13, 15, 18, 24])
def test_bounds_of_a_batch_with_and_without_room_for_its_records(pkg, mb):
    """Under a small cap the bounds come from the finished tile instead of the
    batch's own records; the bytes are the same."""
    V, vo, F, fo = pkg.tdp.gen_meshes(2, 1, seed=3, which="vessels")
    meshes = [(V[vo[i]:vo[i + 1]], F[fo[i]:fo[i + 1]]) for i in range(2)]
    with pkg.Context(0, budget_bytes=mb << 20) as small:
        raw, info = small.raw_from_meshes(V, vo, F, fo, voxel_size=100)
        raw = np.array(raw)
    np.testing.assert_array_equal(raw, oracle_bounds(oracle_prep(meshes)))
    assert info["batches"] == 1
