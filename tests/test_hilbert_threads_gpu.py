"""Analytic signals of different lengths from several threads at once: the kernels' shared-memory limits
are per kernel, not per call, so no thread may lower another's."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from oracle import analytic
from tests import _helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames", [1, 2])  # in place, out of place
def test_lengths_side_by_side(cuda, frames):
    import torch

    from mach_b200 import ingest

    x = {n: np.random.default_rng(n).normal(size=(1, 4, n, frames)).astype(np.float32) for n in (256, 3072, 4096, 6144)}
    want = {n: analytic.analytic_signal(v, axis=2) for n, v in x.items()}
    dev = {n: torch.as_tensor(v, device="cuda") for n, v in x.items()}
    failed = []

    def work(n):
        try:
            for _ in range(300):
                got = ingest.hilbert(dev[n], "c64", layout="channel")
            if not H.rel_l2(got.cpu().numpy(), want[n]) <= 1e-5:
                failed.append((n, "wrong"))
        except Exception as err:
            failed.append((n, str(err)))

    threads = [threading.Thread(target=work, args=(n,)) for n in x for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
