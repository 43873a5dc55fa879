"""The in-place analytic-signal kernel against the FP64 oracle: every radix, several column pairs per
CTA, column counts that leave a pair or a group unfinished, both layouts and all storage types.
Tolerance as in test_hilbert_gpu: 1e-5 relative L2 for FP32 transforms."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import analytic
from tests import _helpers as H

pytestmark = pytest.mark.gpu

LENGTHS = [64, 72, 80, 100, 130, 176, 208, 250, 256, 416, 512, 600, 1000, 1536, 2000, 2500, 3072, 4096, 5000, 6144]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("cols", [(1, 1), (3, 1), (5, 7), (2, 33), (16, 40)])
def test_acquisition_layout(cuda, n, cols):
    import torch

    from mach_b200 import ingest

    x = np.random.default_rng(n).normal(size=(n, *cols)).astype(np.float32)
    got = ingest.hilbert(torch.as_tensor(x, device="cuda"), layout="acquisition").cpu().numpy()
    want = analytic.preprocess_signal(x)
    np.testing.assert_array_equal(got.real, want.real.astype(np.float32))
    assert H.rel_l2(got, want) <= 1e-5


@pytest.mark.parametrize("n", [256, 1024, 3328])
@pytest.mark.parametrize("src", ["f32", "f16", "bf16", "i16"])
@pytest.mark.parametrize("layout", ["channel", "acquisition"])
def test_storages_and_misaligned_source(cuda, n, src, layout):
    import torch

    from mach_b200 import ingest

    shape = (2, 9, n, 1) if layout == "channel" else (n, 9, 2)
    x = torch.as_tensor(np.random.default_rng(1).normal(size=shape) * 100)
    x = x.to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "i16": torch.int16}[src])
    flat = torch.zeros(x.numel() + 1, dtype=x.dtype, device="cuda")
    flat[1:] = x.cuda().reshape(-1)
    for sig in (x.cuda(), flat[1:].view(shape)):  # the second one element off every wider alignment
        got = ingest.hilbert(sig, "c64", layout=layout, scale=0.5).cpu().numpy()
        ref = x.float().numpy() * 0.5
        want = analytic.analytic_signal(ref, axis=2) if layout == "channel" else analytic.preprocess_signal(ref)
        assert H.rel_l2(got, want) <= 1e-5
