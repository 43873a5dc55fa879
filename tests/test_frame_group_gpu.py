"""Complex ensembles on groups of 2, 4, 8 and 16 lanes per voxel: every split of the frames into launches,
every storage and interpolation, rows that end inside the image, small grids, and batches."""

from __future__ import annotations

import numpy as np
import pytest

from tests import _helpers as H
from tests.test_kernels_gpu import _workload

pytestmark = pytest.mark.gpu

COMPLEX = ["c64", "cf16", "cbf16", "ci16"]


@pytest.mark.parametrize("storage", COMPLEX)
@pytest.mark.parametrize("interp", [0, 1, 2])
@pytest.mark.parametrize("n_frames", [16, 24, 32, 40, 48, 56, 72, 88, 104, 128, 168, 200])
def test_matches_the_warp_kernel_and_oracle(cuda, storage, interp, n_frames):
    w = _workload(storage, n_frames, interp)
    got, warp = H.gpu_compound(w), H.gpu_compound(w, kernel="warp")
    assert H.rel_l2(got, warp) < 1e-6  # same taps and weights, sums in another order
    assert H.nrms_db(got, H.oracle(w)) < -60


@pytest.mark.parametrize("delay", ["reference", "split"])
@pytest.mark.parametrize("interp", [0, 1, 2])
@pytest.mark.parametrize("n_frames,n_tx", [(16, 1), (40, 2), (64, 5), (136, 2)])
def test_rows_that_end_inside_the_image(cuda, delay, interp, n_frames, n_tx):
    w = H.small("doppler", n_frames=n_frames, n_tx=n_tx, n_samples=500)
    w.params["interp_type"] = interp
    got, warp = H.gpu_compound(w, delay=delay), H.gpu_compound(w, delay=delay, kernel="warp")
    assert np.abs(got).max() > 0
    assert H.rel_l2(got, warp) < 1e-6


@pytest.mark.parametrize("n_x,n_z", [(1, 1), (3, 5), (9, 33), (130, 7)])
@pytest.mark.parametrize("n_frames", [16, 32, 40, 64, 128])
def test_tiling_never_changes_a_sum(cuda, n_x, n_z, n_frames):
    w = H.small("doppler", n_x=n_x, n_z=n_z, n_frames=n_frames, n_elements=40)
    base = H.gpu_compound(w, grid_shape=False)
    for kw in ({"grid_shape": (n_x, 1, n_z)}, {"tile_fast": 1}, {"tile_fast": 16}, {"tile_order": 2}):
        np.testing.assert_array_equal(base, H.gpu_compound(w, **kw))


@pytest.mark.parametrize("n_frames", [16, 32, 40, 48, 72, 128])
@pytest.mark.parametrize("storage", ["c64", "cf16"])
def test_batch_is_bit_identical(cuda, n_frames, storage):
    import torch

    from mach_b200.batch import Batch, Job

    jobs, want = [], []
    for n_x in (8, 13):
        w = H.small("doppler", n_x=n_x, n_frames=n_frames, n_elements=32)
        ch = w.channel if storage == "c64" else torch.view_as_real(w.channel).half()
        w.channel, w.storage = ch.contiguous(), storage
        t = [torch.as_tensor(x, device="cuda") for x in (ch, w.rx_coords_m, w.scan_coords_m, w.tx_wave_arrivals_s)]
        jobs.append(Job(t[0].contiguous(), *t[1:], **{k: w.params[k] for k in H.PARAM_KEYS}))
        want.append(H.gpu_compound(w))
    batch = Batch(jobs)
    batch.run()
    for j, ref in zip(jobs, want):
        np.testing.assert_array_equal(j.out.cpu().numpy(), ref)
    batch.close()
