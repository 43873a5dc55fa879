"""How the planner splits frames: small scans run in one launch of wide frame groups, larger ones in several,
and rows that need a padded copy get one only where that pays.  Whatever it chooses, the image is the warp
kernel's (tolerance of the other chunk kernels' tests: the same taps and weights, sums in another order)."""

from __future__ import annotations

import pytest

from tests import _helpers as H
from tests.test_batch_limits_gpu import _job
from tests.test_kernels_gpu import STORAGES, _workload

pytestmark = pytest.mark.gpu


def _launches(w, **kw):
    from mach_b200 import _cuda_impl as C

    before = C.launch_count()
    got = H.gpu_compound(w, **kw)
    return got, C.launch_count() - before


# (n_x, n_z) just below and above 4096, 8192, 16384, 32768 and 65536 points
SCANS = [(32, 128), (33, 128), (64, 128), (65, 128), (128, 128), (129, 128), (256, 128), (257, 128), (512, 128),
         (513, 128)]


@pytest.mark.parametrize("storage", ["c64", "cf16"])
@pytest.mark.parametrize("n_frames", [24, 40, 48, 72, 104, 136])
@pytest.mark.parametrize("scan", SCANS)
def test_splits_match_the_warp_kernel(cuda, storage, n_frames, scan):
    w, _ = _job(storage, n_frames, 1, n_x=scan[0], n_z=scan[1], n_elements=4, n_samples=300)
    got, launches = _launches(w)
    n = scan[0] * scan[1]
    if n <= 16384 or n_frames in (24, 104) or (n_frames <= 48 and n <= 65536):
        assert launches == 1
    assert H.rel_l2(got, H.gpu_compound(w, kernel="warp")) < 1e-6


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("n_frames", [9, 13, 17, 33])
def test_padded_rows_on_request(cuda, storage, n_frames):
    """A small scan is not worth the copy; asked for, the chunk kernels run on one all the same."""
    w = _workload(storage, n_frames, 1)
    got, launches = _launches(w, kernel="lane_voxel")
    warp = H.gpu_compound(w, kernel="warp")
    assert launches >= 2  # the copy and the gather
    assert H.rel_l2(got, warp) < 1e-6
    auto, launches = _launches(w)
    assert H.rel_l2(auto, warp) < 1e-6
    if storage != "c64" and w.n_vox < w.channel.shape[2]:
        assert launches == 1


@pytest.mark.parametrize("storage,n_frames,scan,copies", [
    ("cf16", 9, (127, 129), False), ("cf16", 9, (128, 128), True), ("cf16", 9, (128, 129), True),
    ("cf16", 17, (23, 26), False), ("cf16", 17, (24, 25), True), ("i16", 9, (127, 129), False),
    ("i16", 9, (128, 128), True),
    ("i16", 17, (64, 127), False), ("i16", 17, (64, 128), True), ("f32", 17, (96, 127), False),
    ("f32", 17, (96, 128), True), ("f32", 11, (128, 128), True), ("c64", 9, (4, 5), True), ("f32", 12, (4, 5), True)])
def test_where_the_copy_pays(cuda, storage, n_frames, scan, copies):
    """Rows of whole 8-byte vectors always get it; up to 15 other frames from 16384 points on, more from a line of
    their type (complex: 2 points per sample, 16-bit real 8192 points, float32 12288)."""
    w, _ = _job(storage, n_frames, 1, n_x=scan[0], n_z=scan[1], n_elements=4, n_samples=300)
    got, launches = _launches(w)
    assert launches == (2 if copies else 1)
    assert H.rel_l2(got, H.gpu_compound(w, kernel="warp")) < 1e-6
