"""Batch jobs at the edges of shared memory: as many transmits as one pass stages (with split delays the
staged words fill 48 KB beside the kernel's own arrays)."""

from __future__ import annotations

import numpy as np
import pytest

from tests import _helpers as H

pytestmark = pytest.mark.gpu


def _job(storage, n_frames, n_tx, n_x=6, n_z=16, n_elements=16, n_samples=600, **kw):
    import torch

    from mach_b200 import workloads as W
    from mach_b200.batch import Job

    w = H.small("doppler", n_x=n_x, n_z=n_z, n_tx=n_tx, n_frames=n_frames, n_elements=n_elements, n_samples=n_samples,
                n_scatterers=20)
    if storage in ("f32", "i16"):
        w.channel, w.storage, w.params["modulation_freq_hz"] = w.channel.real.contiguous(), "f32", 0.0
    w.channel, w.channel_scale = W.as_storage(w, storage)
    w.storage = storage
    return w, Job(channel=w.channel.cuda().contiguous(), rx_coords_m=torch.as_tensor(w.rx_coords_m).cuda(),
                  scan_coords_m=torch.as_tensor(w.scan_coords_m).cuda(),
                  arrivals=torch.as_tensor(w.tx_wave_arrivals_s).cuda(), channel_scale=w.channel_scale,
                  **{k: w.params[k] for k in H.PARAM_KEYS}, **kw)


# n_tx = lanes per voxel x 32: one frame runs 4 lanes, 16 / 32 / 64 / 128 complex frames 2 / 4 / 8 / 16 lanes
@pytest.mark.parametrize("storage,n_frames,n_tx", [
    ("i16", 1, 128), ("i16", 1, 255), ("cf16", 1, 128), ("i16", 3, 32), ("i16", 8, 63), ("i16", 16, 64),
    ("cf16", 5, 32), ("cf16", 24, 32), ("cf16", 16, 64), ("ci16", 32, 128), ("cf16", 64, 256), ("cbf16", 40, 128)])
def test_split_delays_at_the_staging_limit(cuda, storage, n_frames, n_tx):
    from mach_b200.batch import Batch

    w, job = _job(storage, n_frames, n_tx)
    batch = Batch([job])
    try:
        batch.run()
        got = job.out.cpu().numpy()
    finally:
        batch.close()
    alone = H.gpu_compound(w)
    assert np.abs(alone).max() > 0
    np.testing.assert_array_equal(got, alone)
