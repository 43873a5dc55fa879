"""The autotuner times what an untuned call runs, for every frame count, and forgets what it timed on other
kernels; its choice for a frame count that single calls pad still runs in a batch."""

from __future__ import annotations

import numpy as np
import pytest

from mach_b200 import tuning
from tests import _helpers as H


@pytest.mark.parametrize("storage", ["c64", "cf16", "f32", "i16"])
@pytest.mark.parametrize("n_frames", [9, 12, 15, 17, 30, 100])
@pytest.mark.parametrize("grid", [None, (1, 64, 64)])
def test_chunk_kernels_are_candidates_for_every_frame_count(storage, n_frames, grid):
    every = tuning.candidates(storage, n_frames, grid)
    assert any(c["kernel"] == "lane_voxel" for c in every)
    plain = tuning.plain_candidates(storage, n_frames, grid)
    assert all(set(c) == {"kernel"} for c in plain)
    assert {c["kernel"] for c in plain} == {c["kernel"] for c in every}


def test_entries_of_other_kernels_are_not_used(tmp_path, monkeypatch):
    monkeypatch.setenv("MACH_B200_TUNING_CACHE", str(tmp_path / "tuning.json"))
    monkeypatch.setattr(tuning, "_MEMO", {})
    monkeypatch.setattr(tuning, "_LOADED", False)
    monkeypatch.setitem(tuning._DEVICE_NAMES, 0, "NVIDIA B200")
    args = ("c64", 3, 128, 2000, 12, 4096, None, 1)
    now = tuning._key(*args, "NVIDIA B200", "reference")
    monkeypatch.setattr(tuning, "KERNEL_SET", tuning.KERNEL_SET - 1)
    before = tuning._key(*args, "NVIDIA B200", "reference")
    monkeypatch.undo()
    monkeypatch.setenv("MACH_B200_TUNING_CACHE", str(tmp_path / "tuning.json"))
    monkeypatch.setattr(tuning, "_MEMO", {})
    monkeypatch.setattr(tuning, "_LOADED", False)
    monkeypatch.setitem(tuning._DEVICE_NAMES, 0, "NVIDIA B200")
    unversioned = now.rsplit("|k", 1)[0]
    for key in (before, unversioned):
        tuning._store(key, {"kernel": "staged", "ms": 1.0})
    assert tuning.lookup(*args, 0, "auto") is None
    tuning._store(now, {"kernel": "lane_voxel", "ms": 1.0})
    monkeypatch.setattr(tuning, "_LOADED", False)
    assert tuning.lookup(*args, 0, "auto") == {"kernel": "lane_voxel"}


@pytest.mark.gpu
@pytest.mark.parametrize("storage", ["c64", "cf16"])
def test_padded_choice_in_a_batch(cuda, storage):
    from mach_b200.batch import Batch
    from tests.test_batch_limits_gpu import _job

    w, job = _job(storage, 12, 2, tuning={"kernel": "lane_voxel"})
    batch = Batch([job])
    try:
        batch.run()
        got = job.out.cpu().numpy()
    finally:
        batch.close()
    np.testing.assert_array_equal(got, H.gpu_compound(w, kernel="staged"))


@pytest.mark.gpu
def test_tuned_twelve_frames(cuda, tmp_path, monkeypatch):
    import torch

    monkeypatch.setenv("MACH_B200_TUNING_CACHE", str(tmp_path / "tuning.json"))
    monkeypatch.setattr(tuning, "_MEMO", {})
    w = H.small("doppler", n_frames=12, n_tx=2)
    args = [torch.as_tensor(x).cuda() for x in (w.channel, w.rx_coords_m, w.scan_coords_m, w.tx_wave_arrivals_s)]
    best = tuning.tune(*args, **{k: w.params[k] for k in H.PARAM_KEYS})
    assert H.rel_l2(H.gpu_compound(w, **best), H.gpu_compound(w)) < 1e-5
