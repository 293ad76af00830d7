"""LOD preparations of meshes of different sizes in several threads, each with a
context of its own: a kernel's limit of dynamic shared memory is the process's."""
import threading

import numpy as np
import pytest

from test_lodprep import icosphere

pytestmark = pytest.mark.gpu


def test_threads_with_meshes_of_their_own_sizes(pkg):
    meshes = [pkg.tdp.stack_meshes([icosphere(s, 5.0 + s)]) for s in (2, 3, 3, 4, 4, 5)]
    with pkg.Context(0) as c:
        want = [c.raw_from_meshes(*m, voxel_size=100)[0].copy() for m in meshes]
    errors = []

    def work(k):
        try:
            with pkg.Context(0) as c:
                for _ in range(60):
                    np.testing.assert_array_equal(c.raw_from_meshes(*meshes[k], voxel_size=100)[0], want[k])
        except Exception as e:  # noqa: BLE001
            errors.append((k, repr(e)[:300]))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(meshes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
