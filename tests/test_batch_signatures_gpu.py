"""A batch of every kernel signature that complex ensembles have: each storage, interpolation and delay mode,
in frame counts that run as several launches of different kernels."""

from __future__ import annotations

import copy

import numpy as np
import pytest

from tests import _helpers as H
from tests.test_batch_limits_gpu import _job

pytestmark = pytest.mark.gpu


def test_every_signature_of_complex_ensembles(cuda):
    import torch

    from mach_b200.batch import Batch

    pairs = []
    # 128 + 32 + 16, 128 + 64 + 8 and 64 + 32 frames: five kernels (a scan this large is not run in one launch)
    for n_frames in (176, 200, 96):
        for storage in ("c64", "cf16", "cbf16", "ci16"):
            base, first = _job(storage, n_frames, 1, n_x=258, n_z=128, n_elements=2, n_samples=300)
            for interp in (0, 1, 2):
                for delay in ("reference", "split"):
                    w = copy.copy(base)
                    w.params = dict(base.params, interp_type=interp)
                    job = copy.copy(first)
                    job.interp_type, job.delay, job.out = interp, delay, torch.zeros_like(first.out)
                    pairs.append((w, job, delay))
    batch = Batch([j for _, j, _ in pairs])
    try:
        batch.run()
        for w, job, delay in pairs:
            alone = H.gpu_compound(w, delay=delay)
            assert np.abs(alone).max() > 0
            np.testing.assert_array_equal(job.out.cpu().numpy(), alone)
    finally:
        batch.close()
