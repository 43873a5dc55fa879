"""How the planner splits frames: small scans run in one launch of wide frame groups, larger ones in several.
Whatever it chooses, the image is the warp kernel's (tolerance of the other chunk kernels' tests: the same taps and weights, sums in another order)."""

from __future__ import annotations

import pytest

from tests import _helpers as H
from tests.test_batch_limits_gpu import _job

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
