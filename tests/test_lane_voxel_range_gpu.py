"""The voxel-per-lane kernels' transmit loop without range tests against the one with them.

A job whose every point is inside its rows takes the loop without tests; the same job with one
more transmit that lies outside every row takes the loop with tests, and that transmit adds
nothing, so both give the same bits.  Rows that end inside the image mix both loops and are
compared with the FP64 oracle."""

from __future__ import annotations

import numpy as np
import pytest

from tests import _helpers as H
from tests.test_kernels_gpu import STORAGES, _workload

pytestmark = pytest.mark.gpu


def _with_far_transmit(w):
    """A copy of ``w`` with one more transmit, 0.5 s late: past the end of every row."""
    import copy

    import torch

    far = copy.copy(w)
    far.channel = torch.cat([w.channel, w.channel[:1]])
    far.tx_wave_arrivals_s = np.concatenate([w.tx_wave_arrivals_s, np.full_like(w.tx_wave_arrivals_s[:1], 0.5)])
    return far


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("interp", [0, 1, 2])
@pytest.mark.parametrize("n_frames", [1, 3, 16, 24])
@pytest.mark.parametrize("delay", ["reference", "split"])
def test_loop_without_tests_is_bit_identical(cuda, storage, interp, n_frames, delay):
    w = _workload(storage, n_frames, interp)
    far = _with_far_transmit(w)
    for lanes in (1, 2, 4) if n_frames == 1 else (0,):
        kw = dict(kernel="lane_voxel", delay=delay, lanes_per_voxel=lanes)
        a, b = H.gpu_compound(w, **kw), H.gpu_compound(far, **kw)
        assert np.abs(a).max() > 0
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("interp", [0, 1, 2])
@pytest.mark.parametrize("n_frames,n_samples", [(1, 500), (1, 501), (16, 500), (40, 501)])
def test_rows_that_end_inside_the_image(cuda, interp, n_frames, n_samples):
    w = H.small("doppler", n_frames=n_frames, n_samples=n_samples)
    w.params["interp_type"] = interp
    got, want = H.gpu_compound(w, delay="split"), H.oracle(w)
    # nearest: an FP64 tie or edge may fall the other way on single points
    assert H.nrms_db(got, want) < (-50 if interp == 0 else -80)


@pytest.mark.parametrize("dtype", ["float32", "complex64", "float16", "bfloat16"])
@pytest.mark.parametrize("n_frames", [1, 2, 16])
@pytest.mark.parametrize("delay", ["reference", "split"])
def test_unused_tap_is_not_read(cuda, dtype, n_frames, delay):
    """A sample position that is a whole number reads that sample alone: an infinity in the next
    one does not reach the sum.  (Sound speed and sampling rate are powers of two, so the
    positions are exact.)"""
    import torch

    from mach_b200 import experimental

    c, fs, k = 1024.0, float(1 << 20), 100
    dt = getattr(torch, dtype)
    ch = torch.full((2, 1, 300, n_frames), 3.0, device="cuda").to(dt)
    ch[:, :, k + 1] = float("inf")
    z = k * c / fs
    scan = torch.tensor([[0.0, 0.0, z]] * 7, device="cuda")
    out = experimental.beamform(ch, torch.zeros((1, 3), device="cuda"), scan, torch.zeros((2, 7), device="cuda"),
                                rx_start_s=0.0, sampling_freq_hz=fs, f_number=1.0, sound_speed_m_s=c,
                                modulation_freq_hz=0.0, tukey_alpha=0.0, delay=delay)
    want = torch.full((7, n_frames), 6.0, device="cuda").to(out.dtype)
    assert torch.equal(out, want)
