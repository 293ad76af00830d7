"""LOD preparation of meshes whose FP32 squared distances overflow: coordinates
are any finite floats, and the rule's choices are those of the FP64 oracle."""
import numpy as np
import pytest

from test_bounds import oracle_bounds
from test_lodprep import icosphere, oracle_prep

pytestmark = pytest.mark.gpu


def meshes(power):
    out = [icosphere(2, 10.0, (3.0, -5.0, 8.0), 0.05, 1), icosphere(1, 4.0, (-20.0, 1.0, 0.5), 0.1, 2)]
    return [(V * np.float32(2.0 ** power), F) for V, F in out]


@pytest.mark.parametrize("power", [0, 61, 64, 80, 115])
def test_transform(pkg, ctx, power):
    """An object's last 12 bytes: its vertex nearest the box centre, the first where all are infinitely far."""
    for m in meshes(power):
        V, vo, F, fo = pkg.tdp.stack_meshes([m])
        raw, _ = ctx.raw_from_meshes(V, vo, F, fo, voxel_size=40)
        want = oracle_prep([m], voxel_size=40)
        assert raw.size == want.size
        np.testing.assert_array_equal(raw[-12:], want[-12:])


@pytest.mark.parametrize("power", [-100, -40, 0, 40, 58, 60, 61, 62, 63, 64, 66, 80, 100, 115])
@pytest.mark.parametrize("voxel_size", [7, 40])
def test_bounds(pkg, ctx, power, voxel_size):
    """Whole tiles, byte for byte: voxels are left out of a nearest-triangle search by FP32 gaps that may overflow."""
    ms = meshes(power)
    V, vo, F, fo = pkg.tdp.stack_meshes(ms)
    raw, _ = ctx.raw_from_meshes(V, vo, F, fo, voxel_size=voxel_size)
    np.testing.assert_array_equal(raw, oracle_bounds(oracle_prep(ms, voxel_size=voxel_size)))
