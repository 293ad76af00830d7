"""The bounded queue of the LOD loop (csrc/task_queue.cuh) with more entries than
a 32-bit count holds: every place is given once, and the counter never wraps."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
HARNESS = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "csrc/task_queue.cuh"

// w warps take turns, `each` entries a claim, until `entries` were claimed
int main(int, char** v) {
    const unsigned cap = strtoul(v[1], 0, 10), warps = strtoul(v[2], 0, 10), each = strtoul(v[3], 0, 10);
    const uint64_t entries = strtoull(v[4], 0, 10);
    std::vector<uint8_t> used(cap, 0);
    std::vector<tdp::QueueClaims> q(warps);
    unsigned ctr = 0;
    uint64_t given = 0, most = 0, elsewhere = 0;
    for (uint64_t done = 0, w = 0; done < entries; done += each, w = (w + 1) % warps) {
        const unsigned at = q[w].claim(each, cap, [&](unsigned n) { const unsigned x = ctr; ctr += n; return x; });
        if (ctr > most) most = ctr;
        for (unsigned i = 0; i < each; ++i) {
            if (at + i >= cap) { ++elsewhere; continue; }
            if (used[at + i]++) { printf("place %u given twice\n", at + i); return 1; }
            ++given;
        }
    }
    const unsigned there = ctr < cap ? ctr : cap;
    if (given != there || most != ctr || ctr >= (uint64_t)cap + (uint64_t)(warps + 1) * each) {
        printf("counter %u (at most %llu), given %llu\n", ctr, (unsigned long long)most, (unsigned long long)given);
        return 1;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("queue")
    (d / "q.cpp").write_text(HARNESS)
    subprocess.run([shutil.which("g++"), "-O2", "-std=c++17", "-I", str(ROOT / "3dpipe_b200"), "-o", str(d / "q"),
                    str(d / "q.cpp")], check=True)
    return d / "q"


@pytest.mark.parametrize("cap,warps,each,entries", [
    (1 << 17, 4736, 95, (1 << 32) + (1 << 22)),  # wraps a counter that goes on
    (1 << 23, 4736, 64, 1 << 25),
    (1 << 17, 3, 64, 1 << 17),                    # just full
    (1 << 17, 5, 95, 1 << 16),                    # not full
])
def test_places_are_given_once(harness, cap, warps, each, entries):
    r = subprocess.run([str(harness), *map(str, (cap, warps, each, entries))], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
