"""Jobs whose scratch does not fit: the kernels that need none take over (odd frame counts without a padded
copy, power Doppler without the frames' image), what the failed attempt had taken is given back, and the scratch is used again once there
is room.

Each test runs in a process of its own, whose memory pool is still empty, and takes most of the device's free
memory first."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

COMMON = """
import ctypes
import numpy as np, torch
from mach_b200 import _cuda_impl as C, doppler, experimental

lib = C._lib
def pool():
    used, held = ctypes.c_uint64(), ctypes.c_uint64()
    assert lib.mach_b200_pool_stats(ctypes.c_int32(0), ctypes.c_int32(1), ctypes.byref(used), ctypes.byref(held)) == 0
    return held.value

def job(n_rx, n_samples, n_frames, n_x, n_z, n_tx=1):
    g = torch.Generator(device="cuda").manual_seed(1)
    ch = torch.randn((n_tx, n_rx, n_samples, n_frames), dtype=torch.complex64, device="cuda", generator=g)
    rx = torch.zeros((n_rx, 3), device="cuda")
    rx[:, 0] = torch.linspace(-0.01, 0.01, n_rx)
    x, z = torch.meshgrid(torch.linspace(-0.01, 0.01, n_x), torch.linspace(0.005, 0.03, n_z), indexing="ij")
    scan = torch.stack([x.ravel(), torch.zeros(n_x * n_z), z.ravel()], 1).cuda().contiguous()
    arr = (scan[:, 2] / 1540.0).repeat(n_tx, 1).contiguous()
    p = dict(rx_start_s=0.0, sampling_freq_hz=n_samples / 6e-5, f_number=1.5, sound_speed_m_s=1540.0,
             modulation_freq_hz=5e6)
    return (ch, rx, scan, arr), p

def fill(leave):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")

def rel(a, b):
    return float((a - b).abs().norm() / b.abs().norm())
"""

PADDED = """
small, p = job(8, 200, 12, 20, 20)
for k in ("auto", "staged"):
    experimental.beamform(*small, kernel=k, **p)  # loads both routes' kernels
args, p = job(256, 4096, 12, 64, 64, n_tx=3)  # padded copy: 403 MB
n = args[2].shape[0]
want = experimental.beamform(*args, kernel="staged", **p)  # reads the rows as they are
out = torch.zeros((n, 12), dtype=torch.complex64, device="cuda")
full = fill(200 << 20)
held = pool()
for _ in range(2):
    out.zero_()
    experimental.beamform(*args, out, **p)
    assert torch.equal(out, want), rel(out, want)
assert pool() <= held + (64 << 20)
del full
torch.cuda.empty_cache()
again = experimental.beamform(*args, **p)
assert pool() >= 402653184, pool()  # on the padded copy now
assert rel(again, want) < 1e-6 and float(want.abs().max()) > 0
print("done")
"""

# The image of the reference run stays in the pool, so the full device is tested before it.
POWER = """
small, p = job(8, 200, 60, 20, 20)
for k in ("auto", "ensemble"):
    doppler.power_doppler(*small, kernel=k, **p)
doppler.power_doppler(*small, **dict(p, interp_type=2))
args, p = job(8, 256, 60, 1000, 1000)  # image: 480 MB
out = torch.zeros(args[2].shape[0], device="cuda")
full = fill(200 << 20)
held = pool()
doppler.power_doppler(*args, out, **p)  # the ensemble kernel needs no image
assert pool() <= held + (64 << 20)
no_image = out.clone()
try:
    doppler.power_doppler(*args, out, **dict(p, interp_type=2))  # the ensemble kernel has no quadratic taps
    raise AssertionError("an image that does not fit was made")
except RuntimeError as err:
    assert "memory" in str(err), err
del full
torch.cuda.empty_cache()
with_image = doppler.power_doppler(*args, **p)
assert pool() >= 480000000, pool()
assert rel(no_image, with_image) < 1e-5 and float(with_image.max()) > 0
assert float(doppler.power_doppler(*args, **dict(p, interp_type=2)).max()) > 0
print("done")
"""


@pytest.mark.parametrize("name", ["padded", "power"])
def test_scratch_that_does_not_fit(cuda, name):
    code = COMMON + {"padded": PADDED, "power": POWER}[name]
    run = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parents[1], capture_output=True,
                         text=True, timeout=300)
    assert run.returncode == 0 and "done" in run.stdout, run.stdout[-2000:] + run.stderr[-4000:]
