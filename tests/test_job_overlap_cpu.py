"""The batch runner's test for shared buffers (das_overlap.h, compiled with g++) against a test of every pair."""

from __future__ import annotations

import ctypes
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mach_b200" / "csrc"

SOURCE = """
#include "das_overlap.h"
extern "C" int share(int nw, int nr, const long long* v) {  // begin, bytes, job of each range, written ones first
    std::vector<mach_b200::JobRange> w, r;
    for (int i = 0; i < nw + nr; ++i, v += 3)
        mach_b200::add_range(i < nw ? w : r, reinterpret_cast<const void*>(v[0]), v[1], static_cast<unsigned>(v[2]));
    return mach_b200::jobs_share_outputs(w, r);
}
"""


@pytest.fixture(scope="module")
def share(tmp_path_factory):
    d = tmp_path_factory.mktemp("overlap")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "t.cpp"), "-o", str(d / "t.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "t.so"))

    def call(written, read):
        flat = [x for r in written + read for x in r]
        return bool(lib.share(len(written), len(read), (ctypes.c_longlong * max(1, len(flat)))(*flat)))

    return call


def _pairwise(written, read):
    def meet(a, b):
        return a[1] > 0 and b[1] > 0 and a[0] < b[0] + b[1] and b[0] < a[0] + a[1]

    return any(meet(a, b) for i, a in enumerate(written) for b in written[:i]) or any(
        meet(a, b) for a in written for b in read if a[2] != b[2])


def test_edges(share):
    assert not share([], [])
    assert not share([(100, 50, 0)], [(100, 50, 0)])  # its own input: one job, one launch
    assert share([(100, 50, 0)], [(149, 1, 1)])
    assert not share([(100, 50, 0)], [(150, 1, 1), (99, 1, 1), (120, 0, 1)])
    assert not share([(100, 50, 0), (150, 50, 1)], [])  # neighbours
    assert share([(100, 50, 0), (100, 50, 1)], [])  # one image, two jobs
    assert share([(100, 50, 0), (300, 10, 2)], [(90, 400, 2)])  # past its own output, into another job's


@pytest.mark.parametrize("seed", range(40))
def test_against_every_pair(share, seed):
    rng = random.Random(seed)
    hits = 0
    for _ in range(100):
        n = rng.randint(1, 6)
        space = rng.choice([50, 400, 3000])
        written = [(rng.randint(1, space), rng.randint(0, 20), j) for j in range(n)]
        read = [(rng.randint(1, space), rng.randint(0, 30), rng.randrange(n)) for _ in range(rng.randint(0, 8))]
        want = _pairwise(written, read)
        hits += want
        assert share(written, read) == want
    assert 0 < hits < 100
