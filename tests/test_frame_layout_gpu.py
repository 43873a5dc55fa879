"""Multi-frame jobs whose rows are not whole vectors (padded copies) and drop-in calls whose voxel grid
is found on the device."""

from __future__ import annotations

import numpy as np
import pytest

from tests import _helpers as H
from tests.test_kernels_gpu import STORAGES, _workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("n_frames", [9, 15, 16, 17, 24, 31, 33, 70])
def test_any_frame_count_matches_the_warp_kernel_and_oracle(cuda, storage, n_frames):
    w = _workload(storage, n_frames, 1)
    got, warp = H.gpu_compound(w), H.gpu_compound(w, kernel="warp")
    assert H.rel_l2(got, warp) < 1e-6  # same taps and weights, sums in another order
    assert H.nrms_db(got, H.oracle(w)) < -60


@pytest.mark.parametrize("interp", [0, 2])
@pytest.mark.parametrize("storage", ["c64", "ci16", "f32", "i16"])
def test_padded_rows_other_taps(cuda, storage, interp):
    w = _workload(storage, 13, interp)
    assert H.rel_l2(H.gpu_compound(w), H.gpu_compound(w, kernel="warp")) < 1e-6


@pytest.mark.parametrize("n_frames", [12, 16, 24])
def test_misaligned_rows_and_accumulation(cuda, n_frames):
    import torch

    from mach_b200 import experimental

    w = _workload("c64", n_frames, 1)
    p = {k: w.params[k] for k in H.PARAM_KEYS}
    geo = [torch.as_tensor(x, device="cuda") for x in (w.rx_coords_m, w.scan_coords_m, w.tx_wave_arrivals_s)]
    flat = torch.zeros(w.channel.numel() + 1, dtype=torch.complex64, device="cuda")
    flat[1:] = w.channel.cuda().reshape(-1)
    shifted = flat[1:].view(w.channel.shape)  # 8-byte aligned only
    out = torch.full((w.n_vox, n_frames), 1 + 2j, dtype=torch.complex64, device="cuda")
    experimental.beamform(shifted, *geo, out, **p)
    want = H.gpu_compound(w) + np.complex64(1 + 2j)
    assert H.rel_l2(out.cpu().numpy(), want) < 1e-6


@pytest.mark.parametrize("n_x,n_z", [(128, 16), (129, 17), (131, 40), (127, 40), (130, 15), (1, 300)])
@pytest.mark.parametrize("n_frames", [12, 16, 40])
@pytest.mark.parametrize("is_complex", [False, True])
def test_drop_in_call_on_any_grid(cuda, n_x, n_z, n_frames, is_complex):
    """The tiling changes which CTA computes a voxel, never a sum: bit-identical with consecutive voxels."""
    import torch

    import mach_b200
    from mach_b200 import experimental

    w = H.small("doppler", n_x=n_x, n_z=n_z, n_tx=1, n_frames=n_frames, n_elements=32, n_samples=900, n_scatterers=50)
    ch = w.channel.cuda()
    ch = ch if is_complex else ch.real.contiguous()
    rx, scan, arr = (torch.as_tensor(x, device="cuda") for x in (w.rx_coords_m, w.scan_coords_m, w.tx_wave_arrivals_s))
    p = {k: w.params[k] for k in H.PARAM_KEYS}
    got = mach_b200.beamform(ch[0], rx, scan, arr[0], **p)
    want = experimental.beamform(ch, rx, scan, arr, grid_shape=False, kernel="lane_voxel", **p)
    assert float(got.abs().max()) > 0
    assert torch.equal(got, want)


def test_padded_job_under_graph_capture(cuda):
    import torch

    from mach_b200 import experimental

    w = _workload("c64", 13, 1)
    p = {k: w.params[k] for k in H.PARAM_KEYS}
    ch, rx, scan, arr = (torch.as_tensor(x).cuda() for x in (w.channel, w.rx_coords_m, w.scan_coords_m,
                                                             w.tx_wave_arrivals_s))
    out = torch.zeros((w.n_vox, 13), dtype=torch.complex64, device="cuda")
    want = experimental.beamform(ch, rx, scan, arr, **p)  # also warms up
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="relaxed")
        experimental.beamform(ch, rx, scan, arr, out, sync=False, **p)
        graph.capture_end()
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
