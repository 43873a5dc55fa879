"""The launch bound of probed voxel grids (das_tiles.h, compiled with g++): for every extent that the
probe may report, the bound covers the tiles of the voxel-per-lane mapping and is not far above."""

from __future__ import annotations

import ctypes
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mach_b200" / "csrc"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiles")
    src = d / "t.cpp"
    src.write_text('#include "das_tiles.h"\nextern "C" long long tiles(long long n, int v, int w) '
                   '{ return mach_b200::probed_tiles(n, v, w); }\n')
    so = d / "t.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.tiles.restype = ctypes.c_longlong
    lib.tiles.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    return lib


@pytest.mark.parametrize("wf", [1, 2, 4, 8, 16])
def test_bound_covers_every_extent(lib, wf):
    rng = random.Random(wf)
    shapes = [(16, 128), (17, 128), (16, 129), (31, 129), (65536, 128), (16, 100000)]
    shapes += [(rng.randint(16, 700), rng.randint(128, 700)) for _ in range(400)]
    for fast, outer in shapes:
        n = fast * outer
        bound = lib.tiles(n, 128, wf)
        assert -(-n // 128) <= bound
        assert -(-outer * wf // 128) * -(-fast // wf) <= bound
        assert bound <= 2 + 4 * n / 128
