"""Lazily conjugated and negated torch views (a flag on the tensor, not in its memory): inputs are resolved,
an output that is one is refused."""

from __future__ import annotations

import pytest

from tests import _helpers as H


def test_views_of_lazy_tensors():
    import torch

    from mach_b200 import _check, _dlpack

    z = torch.randn(3, 4, 5, dtype=torch.complex64)
    flipped = z.conj()
    assert flipped.is_contiguous() and flipped.data_ptr() == z.data_ptr()
    with pytest.raises(TypeError, match="resolve_conj"):
        _dlpack.view(flipped)
    got = _check.ensure_contiguous(flipped)
    assert not got.is_conj() and torch.equal(got, z.conj_physical())
    negative = z.conj().imag  # the negated imaginary parts, by a flag
    assert negative.is_neg()
    with pytest.raises(TypeError, match="resolve_neg"):
        _dlpack.view(negative)
    got = _check.ensure_contiguous(negative)
    assert got.is_contiguous() and not got.is_neg() and torch.equal(got, -z.imag)
    assert _check.ensure_contiguous(z) is z


@pytest.mark.gpu
@pytest.mark.parametrize("entry", ["drop_in", "compound"])
def test_conjugated_channel_data(cuda, entry):
    import torch

    import mach_b200
    from mach_b200 import experimental

    w = H.small("doppler", n_x=10, n_z=24, n_tx=1, n_frames=3, n_elements=32)
    p = {k: w.params[k] for k in H.PARAM_KEYS}
    ch, rx, scan, arr = (torch.as_tensor(x).cuda() for x in (w.channel, w.rx_coords_m, w.scan_coords_m,
                                                             w.tx_wave_arrivals_s))

    def run(x, out=None):
        if entry == "drop_in":
            return mach_b200.beamform(x[0], rx, scan, arr[0], out, **p)
        return experimental.beamform(x, rx, scan, arr, out, **p)

    assert ch.conj().is_conj()
    want = run(ch.conj_physical())
    assert float((want - run(ch)).abs().max()) > 0
    assert torch.equal(run(ch.conj()), want)
    out = torch.zeros((w.n_vox, 3), dtype=torch.complex64, device="cuda")
    with pytest.raises(ValueError, match="conjugat"):
        run(ch, out.conj())
    assert float(out.abs().max()) == 0


@pytest.mark.gpu
def test_conjugated_batch_buffers(cuda):
    import torch

    from mach_b200.batch import Batch, Job

    w = H.small("doppler", n_x=10, n_z=24, n_tx=1, n_frames=3, n_elements=32)
    p = {k: w.params[k] for k in H.PARAM_KEYS}
    ch, rx, scan, arr = (torch.as_tensor(x).cuda() for x in (w.channel, w.rx_coords_m, w.scan_coords_m,
                                                             w.tx_wave_arrivals_s))
    with pytest.raises(TypeError, match="resolve_conj"):
        Job(channel=ch.conj(), rx_coords_m=rx, scan_coords_m=scan, arrivals=arr, **p)
    out = torch.zeros((w.n_vox, 3), dtype=torch.complex64, device="cuda")
    batch = Batch([Job(channel=ch, rx_coords_m=rx, scan_coords_m=scan, arrivals=arr, out=out.conj(), **p)])
    try:
        with pytest.raises(ValueError, match="Job.out"):
            batch.run()
    finally:
        batch.close()


@pytest.mark.gpu
def test_conjugated_acquisition(cuda):
    import torch

    from mach_b200 import ingest

    z = torch.randn(40, 3, 2, dtype=torch.complex64, device="cuda")
    assert torch.equal(ingest.ingest(z.conj()), ingest.ingest(z.conj_physical()))
    x = z.conj().imag  # negated by a flag
    assert x.is_neg() and torch.equal(ingest.hilbert(x, layout="acquisition"), ingest.hilbert(-z.imag, layout="acquisition"))
    with pytest.raises(ValueError, match="contiguous"):
        ingest.ingest(z, out=torch.empty((2, 3, 40, 1), dtype=torch.complex64, device="cuda").conj())
