"""Jobs of one batch that share buffers run one after the other, in order: two kinds of channel data added
into one image, and a job whose channel data is another job's image."""

from __future__ import annotations

import numpy as np
import pytest

from tests import _helpers as H
from tests.test_batch_limits_gpu import _job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_frames", [1, 3, 24])
def test_one_image_of_several_storages(cuda, n_frames):
    import torch

    from mach_b200.batch import Batch

    pairs = [_job(s, n_frames, n_tx) for s, n_tx in (("c64", 9), ("cf16", 2), ("ci16", 5), ("cbf16", 1))]
    out = torch.zeros_like(pairs[0][1].out)
    for _, job in pairs:
        job.out, job.accumulate = out, True
    want = np.zeros(out.shape, np.complex64)
    for w, _ in pairs:
        want = want + H.gpu_compound(w)
    batch = Batch([j for _, j in pairs])
    try:
        for _ in range(50):
            out.zero_()
            batch.run(sync=False)
            np.testing.assert_array_equal(out.cpu().numpy(), want)
    finally:
        batch.close()


def test_a_job_that_reads_another_jobs_image(cuda):
    import torch

    from mach_b200.batch import Batch

    w1, first = _job("c64", 1, 3)
    w2, second = _job("c64", 1, 1)
    first.interp_type = 0
    rows = w2.channel.shape[1] * w2.channel.shape[2]
    again = -(-rows // w1.n_vox)  # the first image, as often as fills the second job's channel data
    scan = first.scan_coords_m.repeat(again, 1)
    first.scan_coords_m, first.arrivals, first.grid_shape = scan, first.arrivals.repeat(1, again), False
    first.out = torch.zeros((scan.shape[0], 1), dtype=torch.complex64, device="cuda")
    batch = Batch([first])
    batch.run()
    batch.close()
    image = first.out.clone()
    second.channel = image.reshape(-1)[:rows].view(w2.channel.shape).clone()
    batch = Batch([second])
    batch.run()
    batch.close()
    want = second.out.clone()
    assert float(want.abs().max()) > 0
    second.channel = first.out.reshape(-1)[:rows].view(w2.channel.shape)
    batch = Batch([first, second])
    try:
        for _ in range(20):
            first.out.zero_()
            second.out.zero_()
            batch.run(sync=False)
            assert torch.equal(first.out, image) and torch.equal(second.out, want)
    finally:
        batch.close()
