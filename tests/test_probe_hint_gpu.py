"""A grid hint together with MACH_B200_FLAG_PROBE_GRID: the launches of one job tile by the same grid, so
every frame of every voxel is written (33 to 48 frames of a large scan run as several launches of
different tile widths)."""

from __future__ import annotations

import numpy as np
import pytest

from tests import _helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["cf16", "c64"])
@pytest.mark.parametrize("hint", [(660, 50, 2), (660, 25, 4), (330, 50, 4), (660, 1, 100), (1, 1, 1)])
@pytest.mark.parametrize("tile_fast", [0, 16])
def test_hint_beside_the_probe_flag(cuda, storage, hint, tile_fast):
    import torch

    from mach_b200 import _cuda_impl as C
    from mach_b200 import _dlpack
    from mach_b200 import workloads as W

    w = H.small("doppler", n_x=660, n_z=100, n_tx=1, n_frames=40, n_elements=8, n_samples=900, n_scatterers=50)
    ch, scale = W.as_storage(w, storage)
    dev = [x.to("cuda").contiguous() for x in (ch, *map(torch.as_tensor, (w.rx_coords_m, w.scan_coords_m,
                                                                          w.tx_wave_arrivals_s)))]
    views = [_dlpack.view(x) for x in dev]
    kw = dict(n_tx=1, n_rx=8, n_samples=900, n_vox=w.n_vox, n_frames=40, channel_scale=scale,
              **{k: w.params[k] for k in H.PARAM_KEYS})
    flags = C.FLAG_OVERWRITE | C.FLAG_SPLIT_DELAY

    def run(extra, **knobs):
        out = torch.full((w.n_vox, 40), complex("nan"), dtype=torch.complex64, device="cuda")
        o = C.make_options(flags | extra, **knobs)
        C.beamform_compound(views[0], storage, *views[1:], _dlpack.view(out), options=o, **kw)
        return out.cpu().numpy()

    want = run(0)
    got = run(C.FLAG_PROBE_GRID, grid_shape=hint, tile_fast=tile_fast)
    assert np.abs(want).max() > 0
    np.testing.assert_array_equal(got, want)  # neither hint nor probe changes a sum
