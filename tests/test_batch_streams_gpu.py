"""Side streams of batches: made once per device and lent out, not per batch; batches on several threads and
streams, and captured ones whose streams are in use by the open capture, give the images of single calls."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from tests import _helpers as H
from tests.test_batch_limits_gpu import _job

pytestmark = pytest.mark.gpu


def _pairs():
    return [_job(s, f, 2) for s, f in (("c64", 1), ("cf16", 3), ("i16", 1), ("f32", 2), ("c64", 24))]


def _stream_id() -> int:
    from cuda.bindings import runtime

    err, stream = runtime.cudaStreamCreate()
    assert err == 0
    err, number = runtime.cudaStreamGetId(stream)
    assert err == 0
    runtime.cudaStreamDestroy(stream)
    return number


def test_batches_make_no_streams_of_their_own(cuda):
    from mach_b200.batch import Batch

    jobs = [j for _, j in _pairs()]
    first = _stream_id()
    step = _stream_id() - first  # how far one stream moves the numbers
    assert step > 0
    before = _stream_id()
    for _ in range(40):
        batch = Batch(jobs)
        batch.run()
        batch.close()
    assert _stream_id() - before <= 8 * step  # three per batch were 120


def test_threads_and_streams(cuda):
    import torch

    from mach_b200.batch import Batch

    sets = [_pairs() for _ in range(4)]
    want = [H.gpu_compound(w) for w, _ in sets[0]]
    failed = []

    def work(pairs, priority):
        try:
            stream = torch.cuda.Stream(priority=priority)
            batch = Batch([j for _, j in pairs])
            for k in range(40):
                batch.run(sync=k % 3 == 0, stream=stream)
            stream.synchronize()
            for (_, j), x in zip(pairs, want):
                if not np.array_equal(j.out.cpu().numpy(), x):
                    failed.append("wrong image")
            batch.close()
        except Exception as err:
            failed.append(repr(err))

    threads = [threading.Thread(target=work, args=(p, -(i % 2))) for i, p in enumerate(sets)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def test_runs_beside_an_open_capture(cuda):
    import torch

    from mach_b200.batch import Batch

    captured, eager = _pairs(), _pairs()
    want = [H.gpu_compound(w) for w, _ in captured]
    a, b = Batch([j for _, j in captured]), Batch([j for _, j in eager])
    a.run()
    b.run()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _, j in captured + eager:
        j.out.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="relaxed")
        a.run(sync=False, stream=side)  # its side streams belong to the capture now
        b.run(sync=False, stream=other)
        graph.capture_end()
    other.synchronize()
    for (_, j), x in zip(eager, want):
        np.testing.assert_array_equal(j.out.cpu().numpy(), x)
    assert all(float(j.out.abs().max()) == 0 for _, j in captured)
    graph.replay()
    b.run()
    torch.cuda.synchronize()
    for (_, j), x in zip(captured, want):
        np.testing.assert_array_equal(j.out.cpu().numpy(), x)
    del graph
    a.close()
    b.close()
