"""The in-place analytic signal on lengths that bring the radices 3, 6, 7 and 8 to the first, middle and last
stages (those of test_hilbert_cols_gpu never have them), against the FP64 oracle.  Tolerance as there."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import analytic
from tests import _helpers as H

pytestmark = pytest.mark.gpu

# 10 3 3, 12 6 3, 16 8 7, 8 11, 8 13, 16 8, 8 7 7, 16 7 4, 16 10 4, 16 11 7, 10 10 7 2, 16 16 8, 16 7 7 3, 16 12 7 2,
# 16 7 7 4 and 16 7 7 7: with the others every radix of the kernel in each stage that a plan gives it
LENGTHS = [90, 216, 896, 88, 104, 128, 392, 448, 640, 1232, 1400, 2048, 2352, 2688, 3136, 5488]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("layout", ["channel", "acquisition"])
@pytest.mark.parametrize("cols", [(1, 3), (5, 7)])
def test_lengths(cuda, n, layout, cols):
    import torch

    from mach_b200 import ingest

    shape = (*cols, n, 1) if layout == "channel" else (n, *cols)
    x = np.random.default_rng(n).normal(size=shape).astype(np.float32)
    got = ingest.hilbert(torch.as_tensor(x, device="cuda"), layout=layout).cpu().numpy()
    want = analytic.analytic_signal(x, axis=2) if layout == "channel" else analytic.preprocess_signal(x)
    assert H.rel_l2(got, want) <= 1e-5
