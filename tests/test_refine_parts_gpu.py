"""Refine batches cut into parts: at the part's size and around it, with empty
sides and under a memory cap, the same bits as the eager refine of whole pairs
(configuration 2).  A pair with a coordinate that is not finite has no defined
result (what its bounds drop depends on the configuration); a batch with one is
refined whole, and its other pairs are not touched by it."""
import numpy as np
import pytest

from test_refine_gpu import make_batch

pytestmark = pytest.mark.gpu


def both(c, tri, hd, osz):
    out = []
    for cfg in (2, 0):
        c.set_refine_config(cfg)
        out.append(c.refine_batch(tri, hd, osz, form=1))
    c.set_refine_config(0)
    return out


@pytest.mark.parametrize("sizes", [(1, 1), (1, 34), (31, 33), (32, 32), (33, 33), (63, 65), (64, 64), (100, 130), (1, 700)])
@pytest.mark.parametrize("pairs", [1, 7, 300])
def test_parts_give_the_bits_of_whole_pairs(pkg, sizes, pairs):
    rng = np.random.default_rng(pairs + sizes[1])
    tri, hd, osz = make_batch(rng, pairs if sizes[1] < 700 else min(pairs, 20), sizes=sizes)
    finite = np.ones(len(osz), bool)
    if len(osz) > 5:
        osz[2, 1] = 0
        osz[3, 3] = 0
    with pkg.Context(0) as c:
        for data in (hd, None):
            a, b = both(c, tri, data, osz)
            np.testing.assert_array_equal(a, b)
        if len(osz) > 5:
            tri[int(osz[4, 2])] = np.nan
            tri[int(osz[5, 0])] = np.inf
            finite[4:6] = False
            a, b = both(c, tri, hd, osz)
            assert c.stats()["refine_items"] == len(osz)
            np.testing.assert_array_equal(a[finite], b[finite])
            for k in (4, 5):  # whole, as when the batch is that pair alone
                np.testing.assert_array_equal(b[k], c.refine_batch(tri, hd, osz[k:k + 1], form=1)[0])


def test_no_room_for_the_parts(pkg):
    rng = np.random.default_rng(5)
    tri, hd, osz = make_batch(rng, 2000, sizes=(60, 130))
    least = len(tri) * (9 + 2 + 12) * 4 + len(osz) * 32
    with pkg.Context(0) as c:
        want = c.refine_batch(tri, hd, osz, form=1)
    seen = set()
    for extra in range(0, 12 << 20, 256 << 10):
        with pkg.Context(0, budget_bytes=least + extra) as c:
            try:
                got = c.refine_batch(tri, hd, osz, form=1)
            except pkg.TdpError:
                continue
            np.testing.assert_array_equal(got, want)
            seen.add(c.stats()["kernel_launches"])
    assert seen == {2, 3}
