"""A batch of every kernel signature that complex ensembles have: each storage, interpolation and delay mode,
in frame counts that run as several launches of different kernels."""

from __future__ import annotations

import numpy as np
import pytest

from tests import _helpers as H
from tests.test_batch_limits_gpu import _job

pytestmark = pytest.mark.gpu


def test_every_signature_of_complex_ensembles(cuda):
    from mach_b200.batch import Batch

    pairs = []
    for n_frames in (176, 200, 48):  # 128 + 32 + 16, 128 + 64 + 8, 32 + 16 frames: five kernels each
        for storage in ("c64", "cf16", "cbf16", "ci16"):
            for interp in (0, 1, 2):
                for delay in ("reference", "split"):
                    w, job = _job(storage, n_frames, 1, delay=delay)
                    job.interp_type = w.params["interp_type"] = interp
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
