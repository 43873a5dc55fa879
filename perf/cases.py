"""Performance cases of the beamformer: what a user has it do, through its public entry points.

``listed()`` gives fixed cases, ``draw(rng)`` more of the same ranges; ``prepare`` makes a
program's arrays on the GPU, ``run`` is one pass through the public call, ``work`` the bytes and
operations that the pass cannot do without, and ``exact`` the same result in 64 bits from plain
torch.

A case is a dict.  ``path`` is the entry point:

* ``bmode``    -- ``mach_b200.beamform``: one transmit, float32 RF or complex64 IQ;
* ``compound`` -- ``mach_b200.experimental.beamform``: all transmits, any storage;
* ``power``    -- ``mach_b200.doppler.power_doppler``: the power image of an ensemble;
* ``rf2iq``    -- ``mach_b200.ingest.preprocess_signal``: acquisition-order RF to IQ;
* ``batch``    -- ``mach_b200.batch.Batch``: a mix of jobs in one call.

Channel data are echoes of scatterers (a static and a moving group) of a two-cycle pulse at
their exact round-trip delays, with noise, stored as the case's storage type.
"""

from __future__ import annotations

import math

import torch

from mach_b200 import batch as mb_batch
from mach_b200 import beamform, doppler, experimental, ingest, workloads

SOUND_SPEED = 1540.0
PITCH = 0.3e-3
COMPLEX = ("c64", "cf16", "cbf16", "ci16")
SAMPLE_BYTES = {"f32": 4, "c64": 8, "f16": 2, "cf16": 4, "bf16": 2, "cbf16": 4, "i16": 2, "ci16": 4}

# transducers: centre frequency, sampling frequency (Hz)
PROBES = {"linear": (5.208e6, 20.832e6), "doppler": (5.0e6, 20.0e6), "matrix": (3.0e6, 12.0e6)}


def _case(name, path, probe, *, el, tx, ns, nf, nx, nz, ny=1, x=19.0, z0=5.0, z1=45.0, storage="f32", interp=1,
          f_number=1.5, alpha=0.5, delay="auto"):
    """``el`` elements (a matrix probe: per side), ``nx`` x ``ny`` x ``nz`` points over
    +-``x`` mm and ``z0``..``z1`` mm."""
    c = {"path": path, "probe": probe, "el": el, "tx": tx, "ns": ns, "nf": nf, "nx": nx, "ny": ny, "nz": nz, "x": x,
         "z0": z0, "z1": z1, "storage": storage, "interp": interp, "f_number": f_number, "alpha": alpha,
         "delay": delay}
    return ({"name": name} | c) if name else c


def listed():
    return [
        # the smallest call: a live preview frame of a small array, where the launch and the host count
        _case("preview_f32", "bmode", "linear", el=64, tx=1, ns=1024, nf=1, nx=96, nz=128, x=9.0, z1=32.0),
        # an ordinary B-mode frame: one plane wave, 128 channels, Hann apodisation
        _case("plain2d_f32", "bmode", "linear", el=128, tx=1, ns=2048, nf=1, nx=256, nz=256, alpha=1.0),
        # the drop-in single-transmit call on an ensemble, as code written for mach's loop over transmits makes it
        _case("ensemble_c64", "bmode", "doppler", el=128, tx=1, ns=1024, nf=64, nx=256, nz=256, x=16.0, z0=4.0,
              z1=36.0, storage="c64", f_number=1.0, alpha=0.0),
        # plane-wave compounding of a high-quality B-mode frame
        _case("compound_c64", "compound", "linear", el=128, tx=75, ns=3328, nf=1, nx=512, nz=512, x=20.0, z1=55.0,
              storage="c64", interp=2, f_number=1.75),
        # fast compounding on an odd grid, IQ kept as FP16 pairs with the default (split) delays
        _case("compound_cf16", "compound", "linear", el=128, tx=11, ns=2001, nf=1, nx=301, nz=397, storage="cf16"),
        # colour Doppler: a short packet at a few angles
        _case("color_c64", "compound", "doppler", el=128, tx=3, ns=1024, nf=12, nx=192, nz=320, x=16.0, z0=4.0,
              z1=36.0, storage="c64", f_number=1.2),
        # ultrafast Doppler: a long ensemble, single precision
        _case("doppler_c64", "compound", "doppler", el=128, tx=5, ns=1024, nf=200, nx=256, nz=256, x=16.0, z0=4.0,
              z1=36.0, storage="c64", f_number=1.0, alpha=0.0),
        # power Doppler of the same ensemble kept as FP16 pairs
        _case("power_cf16", "power", "doppler", el=128, tx=5, ns=1024, nf=200, nx=256, nz=256, x=16.0, z0=4.0,
              z1=36.0, storage="cf16", f_number=1.0, alpha=0.0),
        # one 3-D volume from a 1024-element matrix array, ADC samples, default delays
        _case("volume_i16", "compound", "matrix", el=32, tx=9, ns=2048, nf=1, nx=128, ny=128, nz=128, x=10.0,
              storage="i16", f_number=1.0),
        # the largest: a 16-frame 3-D acquisition with the reference's delay arithmetic
        _case("volume16_i16", "compound", "matrix", el=32, tx=9, ns=2048, nf=16, nx=128, ny=128, nz=128, x=10.0,
              storage="i16", f_number=1.0, delay="reference"),
        # front end: acquisition-order RF of the compounding frame to IQ in the beamformer's layout
        _case("rf2iq_f32", "rf2iq", "linear", el=128, tx=75, ns=3328, nf=1, nx=0, nz=0),
        # serving: a wave of mixed requests (plain 2-D, compounding, 32-frame Doppler, 3-D), FP16 storage
        _case("batch_f16", "batch", "linear", el=128, tx=1, ns=2048, nf=1, nx=256, nz=256, storage="f16", alpha=1.0),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("bmode", "bmode_frames", "compound", "color", "doppler", "power", "volume", "rf2iq", "batch"))
    grid = {"nx": log(64, 400), "nz": log(96, 500)}
    el = rng.choice((64, 96, 128, 192))
    f_number, alpha = rng.choice((1.0, 1.2, 1.5, 1.75)), rng.choice((0.0, 0.5, 1.0))
    if kind == "bmode":
        return _case("", "bmode", "linear", el=el, tx=1, ns=log(1000, 3400), nf=1, **grid,
                     storage=rng.choice(("f32", "c64")), interp=rng.choice((0, 1, 2)), f_number=f_number, alpha=alpha)
    if kind == "bmode_frames":
        return _case("", "bmode", "doppler", el=el, tx=1, ns=log(900, 2000), nf=log(9, 128), **grid, x=16.0, z0=4.0,
                     z1=36.0, storage=rng.choice(("f32", "c64")), f_number=f_number, alpha=alpha)
    if kind == "compound":
        return _case("", "compound", "linear", el=el, tx=log(3, 75), ns=log(1400, 3400), nf=1, **grid, x=20.0,
                     z1=50.0, storage=rng.choice(("f32", "c64", "cf16", "cbf16", "ci16")),
                     interp=rng.choice((1, 2)), f_number=f_number, alpha=alpha)
    if kind == "color":
        return _case("", "compound", "doppler", el=el, tx=log(1, 5), ns=log(900, 2000), nf=log(6, 24), **grid, x=16.0,
                     z0=4.0, z1=36.0, storage=rng.choice(("c64", "cf16", "ci16")), f_number=f_number, alpha=alpha)
    if kind in ("doppler", "power"):
        return _case("", "compound" if kind == "doppler" else "power", "doppler", el=el, tx=log(2, 7),
                     ns=log(900, 1400), nf=8 * log(5, 25) + rng.choice((0, 0, 0, 2, 4, 5)), nx=log(96, 256),
                     nz=log(128, 256), x=16.0, z0=4.0, z1=36.0,
                     storage=rng.choice(("c64", "c64", "cf16", "ci16")), f_number=f_number, alpha=alpha)
    if kind == "volume":
        side = log(40, 100)
        return _case("", "compound", "matrix", el=rng.choice((16, 32)), tx=log(2, 9), ns=log(1500, 2048),
                     nf=rng.choice((1, 1, 4, 16, 16)), nx=side, ny=log(40, 100), nz=log(48, 128), x=10.0,
                     storage=rng.choice(("i16", "i16", "f32", "f16")), f_number=1.0,
                     delay=rng.choice(("auto", "reference")))
    if kind == "rf2iq":
        ns = rng.choice((1024, 1536, 2000, 2048, 2500, 3072, 3328))
        return _case("", "rf2iq", "linear", el=el, tx=log(3, 75), ns=ns, nf=1, nx=0, nz=0,
                     storage=rng.choice(("f32", "f32", "i16")))
    return _case("", "batch", "linear", el=el, tx=1, ns=log(1400, 3000), nf=1, nx=log(96, 300), nz=log(96, 300),
                 storage="f16", alpha=alpha)


# ----------------------------------------------------------------------------- geometry and echoes


def _jobs(case):
    """The beamforming jobs of a case: itself, or the mix that a batch stands for."""
    if case["path"] != "batch":
        return [case]
    nx, nz, ns = case["nx"], case["nz"], case["ns"]
    return [
        case,
        _case("", "compound", "linear", el=case["el"], tx=15, ns=ns, nf=1, nx=nx + 31, nz=nz, x=20.0, storage="cf16",
              interp=2, f_number=1.75),
        dict(case, alpha=0.5),
        _case("", "compound", "doppler", el=case["el"], tx=3, ns=1024, nf=32, nx=nx, nz=nz // 2, x=16.0, z0=4.0,
              z1=36.0, storage="cf16", f_number=1.0, alpha=0.0),
        _case("", "compound", "matrix", el=16, tx=4, ns=1600, nf=1, nx=40, ny=40, nz=64, x=10.0, storage="f16",
              f_number=1.0),
    ]


def _device():
    return torch.device("cuda")


def _geometry(case):
    """Float64 element positions, scan points (z contiguous) and the transmit delay function."""
    dev = _device()
    if case["probe"] == "matrix":
        rx = torch.as_tensor(workloads.matrix_array(case["el"], PITCH), device=dev)
    else:
        rx = torch.as_tensor(workloads.linear_array(case["el"], PITCH), device=dev)
    half = case["x"] * 1e-3
    xs = torch.linspace(-half, half, max(1, case["nx"]), dtype=torch.float64, device=dev)
    ys = torch.linspace(-half, half, case["ny"], dtype=torch.float64, device=dev) if case["ny"] > 1 else xs.new_zeros(1)
    zs = torch.linspace(case["z0"] * 1e-3, case["z1"] * 1e-3, max(1, case["nz"]), dtype=torch.float64, device=dev)
    scan = torch.stack(torch.meshgrid(xs, ys, zs, indexing="ij"), dim=-1).reshape(-1, 3)
    n = case["tx"]
    if case["probe"] == "matrix":  # diverging waves from virtual sources 10 mm behind the array
        src = torch.zeros((n, 3), dtype=torch.float64, device=dev)
        k = torch.arange(n, device=dev)
        src[:, 0] = (k % 3 - 1) * 3e-3
        src[:, 1] = (torch.div(k, 3, rounding_mode="floor") % 3 - 1) * 3e-3
        src[:, 2] = -10e-3

        def delay(p):
            return (torch.cdist(src, p) - torch.linalg.vector_norm(src, dim=1)[:, None]) / SOUND_SPEED
    else:  # plane waves
        top = 16.0 if case["probe"] == "linear" else 4.0
        ang = torch.deg2rad(torch.linspace(-top, top, n, dtype=torch.float64, device=dev)) if n > 1 else scan.new_zeros(1)
        d = torch.stack([torch.sin(ang), torch.zeros_like(ang), torch.cos(ang)], dim=-1)

        def delay(p):
            return d @ p.T / SOUND_SPEED
    return rx, scan, delay


def _echoes(case, rx, delay, gen, n_scatterers):
    """[n_tx, n_rx, n_samples] echoes of random scatterers: RF, or IQ at baseband."""
    dev = _device()
    f0, fs = PROBES[case["probe"]]
    iq = case["storage"] in COMPLEX
    n_tx, n_rx, ns = case["tx"], rx.shape[0], case["ns"]
    lim = max(case["x"], 9.0) * 1e-3
    pos = torch.rand((n_scatterers, 3), generator=gen, device=dev, dtype=torch.float64) * 2 - 1
    pos[:, 0] *= lim
    pos[:, 1] = pos[:, 1] * lim if case["probe"] == "matrix" else 0.0
    pos[:, 2] = (case["z0"] + (pos[:, 2] + 1) / 2 * (case["z1"] - case["z0"])) * 1e-3
    amp = torch.randn(n_scatterers, generator=gen, device=dev, dtype=torch.float64)
    sigma = 0.5 / f0
    half = int(math.ceil(3.0 * sigma * fs))
    taps = torch.arange(-half, half + 1, device=dev, dtype=torch.float64)
    t_rx = torch.cdist(rx, pos) / SOUND_SPEED
    t_tx = delay(pos)
    # sums in fixed point, so that the order of the atomic adds does not show
    parts = 2 if iq else 1
    out = torch.zeros((n_tx, n_rx * ns, parts), dtype=torch.int64, device=dev)
    rows = torch.arange(n_rx, device=dev)[:, None, None] * ns
    for t in range(n_tx):
        tau = t_tx[t] + t_rx
        centre = torch.floor(tau * fs)
        idx = centre[..., None] + taps
        dt = idx / fs - tau[..., None]
        env = amp[:, None] * torch.exp(-0.5 * (dt / sigma) ** 2)
        if iq:
            val = 0.5 * env * torch.exp(-2j * math.pi * f0 * tau)[..., None]
        else:
            val = env * torch.cos(2 * math.pi * f0 * dt)
        inside = (idx >= 0) & (idx < ns)
        flat = (rows + idx.long().clamp(0, ns - 1)).reshape(-1)
        val = torch.view_as_real(val) if iq else val[..., None]
        fixed = (torch.where(inside[..., None], val, 0) * 2.0 ** 40).round().long()
        out[t].index_add_(0, flat, fixed.reshape(-1, parts))
    out = (out.double() * 2.0 ** -40).float()
    return (torch.view_as_complex(out) if iq else out[..., 0]).reshape(n_tx, n_rx, ns)


def _channel(case, rx, delay, gen):
    """(channel data as stored, scale): a static and a moving group of scatterers, and noise."""
    dev = _device()
    storage, nf = case["storage"], case["nf"]
    still = _echoes(case, rx, delay, gen, 300)
    move = _echoes(case, rx, delay, gen, 100) if nf > 1 else None
    parts = []
    for t in range(case["tx"]):
        if move is None:
            x = still[t, :, :, None]
        else:
            turn = 0.05 * math.pi * torch.arange(nf, device=dev, dtype=torch.float32)
            turn = torch.polar(torch.ones_like(turn), turn) if still.is_complex() else torch.cos(turn)
            x = still[t, :, :, None] + move[t, :, :, None] * turn
        x = x + 0.02 * torch.randn(x.shape, generator=gen, device=dev, dtype=x.dtype)
        if storage in ("i16", "ci16"):  # 14-bit converter range, a loud echo near full scale
            x = (torch.view_as_real(x) if x.is_complex() else x) * 1500.0
            x = x.round().clamp(-32768, 32767).to(torch.int16)
        elif storage in ("cf16", "cbf16"):
            x = torch.view_as_real(x).to(torch.float16 if storage == "cf16" else torch.bfloat16)
        elif storage in ("f16", "bf16"):
            x = x.to(torch.float16 if storage == "f16" else torch.bfloat16)
        parts.append(x)
    return torch.stack(parts), 1.0 / 1500.0 if storage in ("i16", "ci16") else 1.0


def _params(case):
    f0, fs = PROBES[case["probe"]]
    return {"rx_start_s": 0.0, "sampling_freq_hz": fs, "f_number": case["f_number"], "sound_speed_m_s": SOUND_SPEED,
            "modulation_freq_hz": f0 if case["storage"] in COMPLEX else 0.0, "tukey_alpha": case["alpha"],
            "interp_type": case["interp"]}


def _inputs(case, gen):
    rx, scan, delay = _geometry(case)
    channel, scale = _channel(case, rx, delay, gen)
    return {"channel": channel, "scale": scale, "rx": rx.float(), "scan": scan.float(), "arrivals": delay(scan).float(),
            "params": _params(case), "case": case}


def _acquisition(case, gen):
    """Real RF in acquisition order [n_samples, n_elements, n_waves]."""
    rx, _, delay = _geometry(case)
    channel, _ = _channel(dict(case, nf=1), rx, delay, gen)
    return channel[..., 0].permute(2, 1, 0).contiguous()


def _generator(seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed)
    return gen


# ----------------------------------------------------------------------------- the passes


def prepare(case, seed):
    gen = _generator(seed)
    if case["path"] == "rf2iq":
        return {"path": "rf2iq", "signal": _acquisition(case, gen)}
    jobs = [_inputs(c, gen) for c in _jobs(case)]
    if case["path"] != "batch":
        return jobs[0] | {"path": case["path"]}
    made = [mb_batch.Job(j["channel"], j["rx"], j["scan"], j["arrivals"], channel_scale=j["scale"], **j["params"])
            for j in jobs]
    return {"path": "batch", "batch": mb_batch.Batch(made), "jobs": made}


def run(state):
    path = state["path"]
    if path == "rf2iq":
        return ingest.preprocess_signal(state["signal"], 0.0, storage="c64")
    if path == "batch":
        state["batch"].run()
        return [j.out for j in state["jobs"]]
    channel, rx, scan, arrivals, p = (state[k] for k in ("channel", "rx", "scan", "arrivals", "params"))
    if path == "bmode":
        return beamform(channel[0], rx, scan, arrivals[0], **p)
    call = experimental.beamform if path == "compound" else doppler.power_doppler
    return call(channel, rx, scan, arrivals, channel_scale=state["scale"], delay=state["case"]["delay"], **p)


def _aperture_share(case):
    """Share of the (point, element) pairs inside the aperture, on a coarse copy of the grid."""
    rng_x = [case["x"] * 1e-3 * (2 * (i + 0.5) / 16 - 1) for i in range(16)]
    n_el = case["el"]
    els = [PITCH * (i - (n_el - 1) / 2) for i in range(n_el)]
    inside = total = 0
    for k in range(16):
        r = (case["z0"] + (k + 0.5) / 16 * (case["z1"] - case["z0"])) * 1e-3 / (2 * case["f_number"])
        for x in rng_x:
            if case["probe"] == "matrix":
                ex = sorted((e - x) ** 2 for e in els[:: max(1, n_el // 16)])
                for y in rng_x[::2]:
                    ey = [(e - y) ** 2 for e in els[:: max(1, n_el // 16)]]
                    inside += sum(1 for a in ex for b in ey if a + b <= r * r)
                    total += len(ex) * len(ey)
            else:
                inside += sum(1 for e in els if abs(e - x) <= r)
                total += n_el
    return inside / total


def work(case):
    """Each input read once, the image written once; per point inside the aperture the
    interpolation (linear: 3, quadratic: 5 operations a component) and the weighted sum."""
    if case["path"] == "rf2iq":
        n = case["el"] * case["tx"] * case["ns"]
        return {"bytes": (8.0 + SAMPLE_BYTES[case["storage"]]) * n, "flops": 5.0 * n * math.log2(case["ns"])}
    total_bytes = flops = 0.0
    for c in _jobs(case):
        cplx = c["storage"] in COMPLEX
        n_rx = c["el"] ** 2 if c["probe"] == "matrix" else c["el"]
        n_vox = c["nx"] * c["ny"] * c["nz"]
        total_bytes += c["tx"] * n_rx * c["ns"] * c["nf"] * SAMPLE_BYTES[c["storage"]]
        total_bytes += n_vox * (12 + 4 * c["tx"]) + 12 * n_rx
        total_bytes += n_vox * 4 * (1 if c["path"] == "power" else c["nf"] * (2 if cplx else 1))
        points = n_vox * n_rx * c["tx"] * c["nf"] * _aperture_share(c)
        per = {0: 0, 1: 3, 2: 5}[c["interp"]] * (2 if cplx else 1) + (8 if cplx else 2)
        flops += points * per
    return {"bytes": total_bytes, "flops": flops}


# ----------------------------------------------------------------------------- 64 bits


def _das64(job):
    """Delay-and-sum of one job in 64 bits: the frames [n_scan, n_frames]."""
    c, p = job["case"], job["params"]
    ch = job["channel"]
    if c["storage"] in ("cf16", "cbf16", "ci16"):
        ch = ch.reshape(*ch.shape[:3], -1)  # (I, Q) as two frames each
    elif c["storage"] == "c64":
        ch = torch.view_as_real(ch).reshape(*ch.shape[:3], -1)
    cplx = c["storage"] in COMPLEX
    n_tx, n_rx, ns, cols = ch.shape
    rx, scan, arr = job["rx"].double(), job["scan"].double(), job["arrivals"].double()
    out = torch.zeros((scan.shape[0], c["nf"]), dtype=torch.complex128 if cplx else torch.float64, device=ch.device)
    base = torch.arange(n_rx, device=ch.device) * ns
    step = max(64, min(1 << 16, (1 << 27) // max(1, n_rx * cols)))
    for v0 in range(0, scan.shape[0], step):
        pts = scan[v0:v0 + step]
        d = rx[None] - pts[:, None]
        h2 = d[..., 0] ** 2 + d[..., 1] ** 2
        dist = torch.sqrt(h2 + d[..., 2] ** 2)
        radius = (pts[:, 2] / (2 * c["f_number"]))[:, None]
        weight = (h2 <= radius ** 2).double()
        if c["alpha"] > 0:
            r = torch.sqrt(h2) / radius
            taper = 0.5 - 0.5 * torch.cos(math.pi * (1 - r) / c["alpha"])
            weight = weight * torch.where(r <= 1 - c["alpha"], 1.0, taper)
        weight = weight * job["scale"]
        for t in range(n_tx):
            tau = arr[t, v0:v0 + step, None] + dist / SOUND_SPEED
            s = tau * p["sampling_freq_hz"]
            if c["interp"] == 0:
                taps = [(torch.round(s), 1.0)]
                ok = (s >= -0.5) & (s <= ns - 0.5) & (taps[0][0] < ns)
            elif c["interp"] == 1:
                lo = torch.floor(s)
                ok = (s >= 0) & (s <= ns - 1)
                taps = [(lo, 1 - (s - lo)), (lo + 1, s - lo)]
            else:
                mid = torch.round(s)
                x = s - mid
                ok = (s >= 1) & (s <= ns - 2)
                taps = [(mid - 1, x * (x - 1) / 2), (mid, 1 - x * x), (mid + 1, x * (x + 1) / 2)]
            w = torch.where(ok & (tau >= 0), weight, 0.0)
            if cplx:
                w = torch.polar(w, 2 * math.pi * p["modulation_freq_hz"] * tau)
            rows = ch[t].reshape(n_rx * ns, cols)
            for idx, share in taps:
                at = base + idx.long().clamp(0, ns - 1)
                x = rows[at.reshape(-1)].double().view(*at.shape, cols)
                wt = w * share
                if cplx:
                    re = torch.bmm(wt.real[:, None], x)[:, 0].view(-1, c["nf"], 2)
                    im = torch.bmm(wt.imag[:, None], x)[:, 0].view(-1, c["nf"], 2)
                    out[v0:v0 + step] += torch.complex(re[..., 0] - im[..., 1], re[..., 1] + im[..., 0])
                else:
                    out[v0:v0 + step] += torch.bmm(wt[:, None], x)[:, 0]
    return out


def exact(case, seed):
    gen = _generator(seed)
    if case["path"] == "rf2iq":
        sig = _acquisition(case, gen)
        n = sig.shape[0]
        h = torch.zeros(n, dtype=torch.float64, device=sig.device)
        h[0] = 1
        h[1:(n + 1) // 2] = 2
        if n % 2 == 0:
            h[n // 2] = 1
        out = torch.empty((sig.shape[2], sig.shape[1], n, 1), dtype=torch.complex128, device=sig.device)
        for w in range(sig.shape[2]):
            z = torch.fft.ifft(torch.fft.fft(sig[:, :, w].double(), dim=0) * h[:, None], dim=0)
            out[w, :, :, 0] = z.T
        return out
    got = [_das64(_inputs(c, gen)) for c in _jobs(case)]
    if case["path"] == "power":
        return got[0].abs().square().sum(dim=1)
    return got if case["path"] == "batch" else got[0]
