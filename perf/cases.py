"""The work this framework is used for, as cases that can be timed and checked.

A case is one call that a user's program makes on data it already holds on the GPU:
delay-and-sum of a frame (``das_fast`` or a resident ``Plan`` on channel data in its
storage type, ``das_table_f32`` on das_c's tables, ``DAS.go`` as a whole), an ensemble of
frames, RF demodulation, and the adaptive weights on a kept channel cube.  Sizes are those
of the synthetic workloads in ``ustb_gb300/synth.py`` and of ``bench.py``, with a preview
of odd sizes at the small end.

Channel data is made of point echoes (the Gaussian pulse of the workloads) in band-limited
noise, so sums are partly coherent as in real recordings.  ``exact`` restates every
operation in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

from ustb_gb300 import fast, kernels, postprocess, preprocess
from ustb_gb300.das import DAS
from ustb_gb300.ensemble import Ensemble
from ustb_gb300.enums import Dimension, Precision, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.plan import Plan
from ustb_gb300.uff import ChannelData, LinearScan, LinearScan3D, Point, Probe, SectorScan, Wave

C = 1540.0
BW = 0.6
SCALE16 = 1.0 / 8192.0  # int16 counts of a recording to channel-data units
DIM = {"none": 0, "receive": 1, "transmit": 2, "both": 3}
PRECISION = {"fp32": Precision.fp32, "fp16": Precision.fp16, "bf16": Precision.bf16}
STORED = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}


def _das(kind, **k):
    """A delay-and-sum case; the defaults are a linear array's plane-wave acquisition."""
    case = dict(kind=kind, nx_el=128, ny_el=1, pitch_um=300.0, wave="plane", w=1, span_deg=16.0, l=1024, f0=5e6,
                t0=0.0, frames=1, scan="linear", nx=256, nz=256, ny=1, z0_mm=5.0, z1_mm=50.0, dim="both",
                window="tukey25", f_number=1.7, storage="fp32", complex=True, epilogue=False)
    case.update(k)
    return case


def listed():
    return [
        # the smallest call: a live preview of one RF plane wave on a resident plan, odd sizes
        dict(_das("plan", nx_el=64, l=1111, nx=101, nz=127, z1_mm=30.0, complex=False), name="preview_rf_plan"),
        # a user's first script: DAS().go() on one RF plane wave, tables, analytic signal
        dict(_das("go", l=2048, complex=False), name="go_rf_plane_wave"),
        # coherent plane-wave compounding of IQ data, the headline workload
        dict(_das("fast", w=75, l=1024, t0=6.5e-6, nx=400, nz=400, z0_mm=8.0, z1_mm=40.0), name="cpwc_iq_fast"),
        # the same frame through the drop-in for das_c: single-precision tables in hand
        dict(_das("table", w=75, l=1024, t0=6.5e-6, nx=400, nz=400, z0_mm=8.0, z1_mm=40.0), name="cpwc_iq_table"),
        # cardiac sector of diverging waves, half-precision storage, channels kept for the
        # coherence factor and simplified DMAS
        dict(_das("fast", nx_el=64, pitch_um=220.0, wave="diverging", w=21, span_deg=30.0, l=1536, f0=3e6,
                  scan="sector", nx=256, nz=512, z1_mm=90.0, dim="transmit", storage="fp16", epilogue=True),
             name="dw_sector_factors_fp16"),
        # synthetic transmit aperture, real RF
        dict(_das("fast", wave="sta", w=128, l=2048, nx=300, nz=300, complex=False), name="sta_rf_fast"),
        # volume of a matrix array, half-precision storage: the largest single frame
        dict(_das("fast", nx_el=32, ny_el=32, wave="diverging", w=25, span_deg=15.0, l=1024, f0=4e6, scan="volume",
                  nx=64, ny=64, nz=128, z1_mm=40.0, storage="fp16"), name="matrix_volume_fp16"),
        # high-frame-rate ensemble (Doppler, functional imaging): int16 I/Q straight from the scanner
        dict(_das("ensemble", w=11, span_deg=10.0, l=1536, frames=50, nx=256, nz=512, storage="fp16"),
             name="hfr_ensemble_int16"),
        # RF recording to half-precision IQ, MATLAB class's causal filter
        dict(kind="demod", l=1536, traces=56320, f0=5e6, over=4, decimation=2, zero_phase=False, source="int16",
             storage="fp16", name="demod_int16_fp16"),
        # the Python port's zero-phase filter on single-precision RF
        dict(kind="demod", l=1536, traces=14080, f0=5e6, over=8, decimation=4, zero_phase=True, source="fp32",
             storage="fp32", name="demod_zero_phase_fp32"),
        # the three coherence weights side by side on a kept channel cube
        dict(kind="factors", nz=512, nx=256, k=64, frames=1, m0=4, weights=True, name="coherence_factors_sector"),
        # minimum variance on the same cube (USTB example settings)
        dict(kind="capon", nz=512, nx=256, k=64, frames=1, l_elements=32, k_samples=7, fb=False, f_number=1.7,
             name="capon_sector"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("fast", "fast", "fast", "plan", "table", "table", "go", "ensemble", "demod", "factors", "capon"))
    if kind == "demod":
        over = rng.choice((4, 8))
        decimation = rng.choice((1, 2, 3, 4))
        return dict(kind="demod", l=_log(rng, 400, 4000), traces=_log(rng, 64, 20000), f0=rng.choice((3e6, 5e6)),
                    over=over, decimation=decimation, zero_phase=rng.random() < 0.5,
                    source=rng.choice(("int16", "fp32")), storage=rng.choice(("fp32", "fp16", "bf16")))
    if kind in ("factors", "capon"):
        case = dict(kind=kind, nz=_log(rng, 64, 600), nx=_log(rng, 32, 256), k=_log(rng, 16, 128),
                    frames=rng.choice((1, 1, 2)))
        if kind == "factors":
            case.update(m0=rng.choice((1, 2, 4)), weights=rng.random() < 0.5)
        else:
            case.update(k=min(case["k"], 64), frames=1, l_elements=min(32, max(4, case["k"] // 2)),
                        k_samples=rng.randint(0, 8), fb=rng.random() < 0.5, f_number=rng.choice((0.0, 1.7)))
            case["nx"] = min(case["nx"], 131072 // case["nz"])
        return case
    scan = "linear" if kind in ("go", "ensemble") else rng.choice(("linear", "linear", "linear", "sector", "volume"))
    case = _das(kind, scan=scan, window=rng.choice(("tukey25", "tukey50", "hanning", "hamming", "boxcar")),
                f_number=rng.choice((1.0, 1.4, 1.7)))
    z1 = rng.uniform(20.0, 60.0)
    if scan == "volume":
        n = rng.randint(8, 24)
        case.update(nx_el=n, ny_el=n, wave="diverging", w=rng.choice((1, 4, 9, 16)), span_deg=15.0, f0=4e6,
                    nx=_log(rng, 17, 64), ny=_log(rng, 17, 64), nz=_log(rng, 40, 128))
    elif scan == "sector":
        case.update(nx_el=_log(rng, 32, 96), pitch_um=220.0, wave="diverging", w=_log(rng, 1, 31), span_deg=30.0,
                    f0=3e6, nx=_log(rng, 64, 256), nz=_log(rng, 128, 512))
        z1 = rng.uniform(40.0, 90.0)
    else:
        case.update(nx_el=_log(rng, 32, 192), nx=_log(rng, 64, 400), nz=_log(rng, 64, 512))
        if kind == "ensemble":
            case.update(w=_log(rng, 1, 15), span_deg=10.0, frames=_log(rng, 4, 50), storage=rng.choice(("fp16", "bf16")))
        elif rng.random() < 0.25:
            case.update(wave="sta", w=case["nx_el"])
        else:
            case.update(w=_log(rng, 1, 75))
    # enough samples for the deepest pixel at four samples per period
    case["z1_mm"] = round(z1, 1)
    case["l"] = int(2.3 * z1 * 1e-3 / C * 4 * case["f0"]) + rng.randint(80, 300)
    if kind == "go":
        case.update(w=min(case["w"], 15), nx=min(case["nx"], 256), nz=min(case["nz"], 256), nx_el=min(case["nx_el"], 128))
        case["complex"] = rng.random() < 0.5
        if case["wave"] == "sta":
            case.update(wave="plane")
    elif kind in ("fast", "plan", "table"):
        case["complex"] = case["wave"] != "sta" and (scan == "volume" or rng.random() < 0.75)
        if kind != "table":
            case["storage"] = rng.choice(("fp32", "fp16", "bf16"))
        case["dim"] = rng.choice(("both", "both", "both", "transmit", "receive"))
        if scan == "volume":
            case["dim"] = "both"
        case["epilogue"] = kind != "table" and case["dim"] == "transmit" and case["complex"]
        case["frames"] = rng.choice((1, 1, 1, 2, 3))
    # no dearer than the listed cases of its kind
    most = {"volume": 2.5e9, "sector": 0.4e9, "linear": 1.5e9}[scan] if kind != "go" else 0.3e9
    per = case["nx_el"] * case["ny_el"] * case["w"] * case["nx"] * case["nz"] * case["ny"]
    if kind == "ensemble":
        case["frames"] = max(2, min(case["frames"], int(6e9 / per)))
    elif per * case["frames"] > most and case["frames"] > 1:
        case["frames"] = 1
    if kind != "ensemble" and per > most:
        case["w"] = max(1, int(case["w"] * most / per))
    return case


# ---------------------------------------------------------------------------
# acquisition and scan of a delay-and-sum case
# ---------------------------------------------------------------------------

def _probe(c):
    p = c["pitch_um"] * 1e-6
    return Probe.matrix_array(c["nx_el"], c["ny_el"], p) if c["ny_el"] > 1 else Probe.linear_array(c["nx_el"], p)


def _angles(w, span_deg):
    return np.deg2rad(np.linspace(-span_deg, span_deg, w)) if w > 1 else np.zeros(1)


def _sources(c):
    """Virtual sources [W, 3] of the spherical waves."""
    if c["wave"] == "sta":
        x = _probe(c).x
        x = x[np.linspace(0, x.size - 1, c["w"]).round().astype(int)]
        return np.stack([x, 0 * x, 0 * x], 1)
    d = 10e-3  # behind the array
    if c["scan"] == "volume":
        side = int(math.isqrt(c["w"]))
        az = np.tile(_angles(side, c["span_deg"]), side + 2)[: c["w"]]
        el = np.repeat(_angles(side, c["span_deg"]), side + 2)[: c["w"]]
    else:
        az = _angles(c["w"], c["span_deg"])
        el = 0 * az
    return np.stack([-d * np.sin(az) * np.cos(el), -d * np.sin(el), -d * np.cos(az) * np.cos(el)], 1)


def _sequence(c):
    if c["wave"] == "plane":
        return [Wave.plane(float(a)) for a in _angles(c["w"], c["span_deg"])]
    if c["wave"] == "sta":  # fired by one element: time zero at that element
        return [Wave(source=Point.from_xyz(*map(float, s)), delay=abs(float(s[0])) / C) for s in _sources(c)]
    return [Wave.diverging(tuple(map(float, s))) for s in _sources(c)]


def _scan(c):
    z = np.linspace(c["z0_mm"] * 1e-3, c["z1_mm"] * 1e-3, c["nz"])
    if c["scan"] == "sector":
        return SectorScan(np.deg2rad(np.linspace(-40, 40, c["nx"])), z)
    if c["scan"] == "volume":
        axis = lambda n: np.linspace(-1, 1, n) * 0.15e-3 * n  # noqa: E731
        return LinearScan3D(axis(c["nx"]), z, axis(c["ny"]))
    half = 0.5 * c["nx_el"] * c["pitch_um"] * 1e-6
    return LinearScan(np.linspace(-half, half, c["nx"]), z)


def _receive(c):
    return Apodization(window=Window[c["window"]], f_number=c["f_number"])


def _fd(c):
    return c["f0"] if c["complex"] else 0.0


def _t(a, dev):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)


def _distance(a, b):
    """[A, B] distances, formed without the matrix-product shortcut."""
    return torch.cdist(a, b, compute_mode="donot_use_mm_for_euclid_dist")


def _transmit_tau(c, xyz):
    """[W, P] transmit delays (s) in double."""
    dev = xyz.device
    if c["wave"] == "plane":
        a = _t(_angles(c["w"], c["span_deg"]), dev)[:, None]
        return (xyz[None, :, 2] * torch.cos(a) + xyz[None, :, 0] * torch.sin(a)) / C
    src = _t(_sources(c), dev)
    d = _distance(src, xyz)
    if c["wave"] == "sta":  # |s| / c cancels between the model's offset and the wave's delay
        return d / C
    return (d - src.norm(dim=1, keepdim=True)) / C


def _window64(name, r):
    one, zero = torch.ones_like(r), torch.zeros_like(r)
    if name == "boxcar":
        return torch.where(r <= 0.5, one, zero)
    if name in ("hanning", "hamming"):
        a, b = (0.5, 0.5) if name == "hanning" else (0.53836, 0.46164)
        return torch.where(r <= 0.5, a + b * torch.cos(2 * math.pi * r), zero)
    roll = {"tukey25": 0.25, "tukey50": 0.5, "tukey75": 0.75}[name]
    taper = 0.5 * (1 + torch.cos(2 * math.pi / roll * (r - roll / 2 - 0.5)))
    return torch.where(r <= 0.5 * (1 - roll), one, torch.where(r < 0.5, taper, zero))


def _receive_apodization(c, el, xyz):
    """[n, P] receive weights in double for elements ``el``."""
    z = xyz[:, 2].abs() if c["scan"] != "sector" else xyz.norm(dim=1)
    z = z.clamp(min=1e-3 * c["f_number"], max=10.0 * c["f_number"])  # smallest aperture 1 mm, largest 10 m
    centre = 0.0 if c["scan"] == "sector" else xyz
    dx = (el[:, None, 0] - (centre[None, :, 0] if c["scan"] != "sector" else 0.0)).abs()
    dy = (el[:, None, 1] - (centre[None, :, 1] if c["scan"] != "sector" else 0.0)).abs()
    if c["scan"] == "sector":
        dx, dy = dx.expand(-1, xyz.shape[0]), dy.expand(-1, xyz.shape[0])
    f = c["f_number"]
    return _window64(c["window"], f * dx / z) * _window64(c["window"], f * dy / z)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _generator(seed, dev):
    return torch.Generator(device=dev).manual_seed(int(seed))


def _noise(shape, g, dev):
    """Band-limited complex or real noise along the last dimension (unit-order level)."""
    x = torch.randn(*shape[:-1], shape[-1] + 4, generator=g, device=dev)
    n = shape[-1]
    return (x[..., :n] + 4 * x[..., 1:n + 1] + 6 * x[..., 2:n + 2] + 4 * x[..., 3:n + 3] + x[..., 4:n + 4]) / 8.37


def _channels(c, seed, dev):
    """One recording (F, W, N, L): complex64 I/Q or float32 RF."""
    g = _generator(seed, dev)
    fs, f0, L, F, W = 4 * c["f0"], c["f0"], c["l"], c["frames"], c["w"]
    el = _t(_probe(c).xyz, dev)
    z0, z1 = c["z0_mm"] * 1e-3, c["z1_mm"] * 1e-3
    u = torch.rand(16, 4, generator=g, device=dev, dtype=torch.float64)
    pts = torch.stack([(u[:, 0] - 0.5) * 0.6 * z1, (u[:, 1] - 0.5) * 0.3 * z1 * (c["ny_el"] > 1),
                       z0 + u[:, 2] * (z1 - z0)], 1)
    tau = _transmit_tau(c, pts).t()[:, :, None] + (_distance(pts, el) / C)[:, None, :]  # [S, W, N]
    n = el.shape[0]
    t = torch.arange(L, device=dev, dtype=torch.float32)
    re = torch.zeros(W, n, L, device=dev)
    im = torch.zeros(W, n, L, device=dev) if c["complex"] else None
    for s in range(pts.shape[0]):
        at = ((tau[s] - c["t0"]) * fs).float()[:, :, None]
        e = t - at
        env = torch.exp(-1.7886 * (e * (BW * f0 / fs)) ** 2)
        amp = float(0.5 + 0.5 * u[s, 3])
        if c["complex"]:
            turn = torch.remainder(-f0 * tau[s], 1.0).float()[:, :, None] * (2 * math.pi)
            re += amp * torch.cos(turn) * env
            im += amp * torch.sin(turn) * env
        else:
            re += amp * env * torch.cos(e * (2 * math.pi * f0 / fs))
    if c["complex"]:
        out = torch.empty(F, W, n, L, dtype=torch.complex64, device=dev)
        for f in range(F):
            out[f] = torch.complex(re + 0.2 * _noise((W, n, L), g, dev), im + 0.2 * _noise((W, n, L), g, dev))
        return out
    carrier = torch.cos(t * (2 * math.pi * f0 / fs))
    return torch.stack([re + 0.2 * _noise((W, n, L), g, dev) * carrier for _ in range(F)])


def _int16_iq(c, seed, dev):
    """An ensemble as the scanner stores it: (F, W, N, L, 2) int16."""
    x = torch.empty(c["frames"], c["w"], c["nx_el"], c["l"], 2, dtype=torch.int16, device=dev)
    one = _channels(dict(c, frames=1), seed, dev)[0]
    g = _generator(seed + 7919, dev)
    for f in range(c["frames"]):
        v = torch.view_as_real(one) + 0.2 * _noise(tuple(one.shape) + (2,), g, dev)
        x[f] = (v / SCALE16).round().clamp(-32768, 32767).to(torch.int16)
    return x


def _stored(c, x):
    """Channel data in its storage type, interleaved re / im for complex data."""
    return (torch.view_as_real(x) if x.is_complex() else x).to(STORED[c["storage"]]).contiguous()


def _pixel_phase(c, scan):
    if not c["complex"]:
        return None
    r = np.asarray(scan.reference_distance, np.float64) * np.ones(scan.N_pixels)
    return np.exp(-4j * math.pi * c["f0"] * r / C)


def _rf(c, seed, dev):
    """RF traces (traces, L) for demodulation: band-limited noise on the carrier."""
    g = _generator(seed, dev)
    fs = c["over"] * c["f0"]
    t = torch.arange(c["l"], device=dev, dtype=torch.float32) * (2 * math.pi * c["f0"] / fs)
    x = torch.empty(c["traces"], c["l"], dtype=torch.int16 if c["source"] == "int16" else torch.float32, device=dev)
    for a in range(0, c["traces"], 16384):
        b = min(a + 16384, c["traces"])
        v = _noise((b - a, c["l"]), g, dev) * torch.cos(t) + _noise((b - a, c["l"]), g, dev) * torch.sin(t)
        x[a:b] = (v * 4096).round().clamp(-32768, 32767).to(torch.int16) if c["source"] == "int16" else v
    return x


def _taps(c):
    fs = c["over"] * c["f0"]
    if c["zero_phase"]:
        return preprocess.python_port_taps(c["f0"], fs, c["l"]).astype(np.float32)
    return preprocess.lowpass_taps(c["f0"], fs).astype(np.float32)


def _cube(c, seed, dev):
    """Kept channel cube (F, 1, K, P): per-pixel coherent part plus noise of varying level."""
    g = _generator(seed, dev)
    F, K, nx, nz = c["frames"], c["k"], c["nx"], c["nz"]

    def field(*shape):
        return torch.complex(_noise(shape, g, dev), _noise(shape, g, dev))

    coherent = field(F, 1, nx, nz)
    level = 0.1 + 2.0 * torch.rand(F, 1, nx, 1, generator=g, device=dev)
    tilt = torch.rand(F, 1, nx, 1, generator=g, device=dev) - 0.5
    k = torch.arange(K, device=dev, dtype=torch.float32)[None, :, None, None] / K
    cube = coherent * torch.polar(torch.ones_like(k * tilt), 2 * math.pi * k * tilt) + level * field(F, K, nx, nz)
    return cube.reshape(F, 1, K, nx * nz).contiguous()


def _cube_weights(c, dev):
    """(K, P) receive weights of a phased array's sector (Tukey 25 %), ones without an F-number."""
    f = c.get("f_number", 1.7)
    if not f:
        return torch.ones(c["k"], c["nx"] * c["nz"], device=dev)
    depth = torch.linspace(5e-3, 90e-3, c["nz"], device=dev, dtype=torch.float64)
    x = (torch.arange(c["k"], device=dev, dtype=torch.float64) - (c["k"] - 1) / 2) * 220e-6
    w = _window64("tukey25", f * x.abs()[:, None] / depth[None, :].clamp(min=1e-3 * f))
    return w.float()[:, None, :].expand(-1, c["nx"], -1).reshape(c["k"], -1).contiguous()


# ---------------------------------------------------------------------------
# prepare, run, work
# ---------------------------------------------------------------------------

def prepare(case, seed):
    c, dev = case, torch.device("cuda", 0)
    kind = c["kind"]
    if kind == "demod":
        return {"case": c, "rf": _rf(c, seed, dev), "taps": _taps(c)}
    if kind == "factors":
        w = _cube_weights(c, dev) if c["weights"] else None
        return {"case": c, "cube": _cube(c, seed, dev), "weights": w,
                "count": (w > 0.16).sum(0).float() if c["weights"] else None}
    if kind == "capon":
        return {"case": c, "cube": _cube(c, seed, dev), "weights": _cube_weights(c, dev)}
    probe, scan, seq, rx = _probe(c), _scan(c), _sequence(c), _receive(c)
    fs = 4 * c["f0"]
    if kind == "go":
        x = _channels(c, seed, dev)
        das = DAS()
        das.channel_data = ChannelData(kernels.to_matlab_order(x), probe, seq, fs, c["t0"], C, _fd(c))
        das.scan = scan
        das.receive_apodization = rx
        das.geometry_fixed = True  # frame after frame of one acquisition
        return {"case": c, "das": das}
    if kind == "table":
        xyz, el = _t(scan.xyz, dev), _t(probe.xyz, dev)
        tx = _transmit_tau(c, xyz).float()
        return {"case": c, "ch": _channels(c, seed, dev), "tx": tx, "tx_apo": torch.ones_like(tx),
                "rx": (_distance(el, xyz) / C).float(), "rx_apo": _receive_apodization(c, el, xyz).float()}
    geom = fast.FastGeometry(probe, scan, seq, fs, c["t0"], _fd(c), C, dev, rx, None, pixel_phase=_pixel_phase(c, scan))
    if kind == "ensemble":
        ens = Ensemble(geom, c["frames"], c["l"], Dimension.both, PRECISION[c["storage"]], SCALE16)
        return {"case": c, "ensemble": ens, "x": _int16_iq(c, seed, dev)}
    state = {"case": c, "ch": _stored(c, _channels(c, seed, dev)), "geom": geom}
    if kind == "plan":
        state["plan"] = Plan(geom, c["l"], PRECISION[c["storage"]], c["complex"], DIM[c["dim"]], c["frames"], c["epilogue"])
    return state


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "plan":
        return state["plan"].execute(state["ch"])
    if kind == "fast":  # flags are read at the end of a stream of frames, as FramePipeline does
        return fast.das_fast(state["ch"], PRECISION[c["storage"]], c["complex"], state["geom"], DIM[c["dim"]],
                             F=c["frames"], epilogue=c["epilogue"], L=c["l"], check=False)
    if kind == "table":
        return kernels.das_table_f32(state["ch"], 4 * c["f0"], c["t0"], state["tx_apo"], state["rx_apo"], state["tx"],
                                     state["rx"], _fd(c), DIM[c["dim"]])
    if kind == "go":
        return state["das"].go().data
    if kind == "ensemble":
        return state["ensemble"].run(state["x"])["cube"]
    if kind == "demod":
        return preprocess.demodulate(state["rf"], c["over"] * c["f0"], 0.0, c["f0"], state["taps"], c["decimation"],
                                     PRECISION[c["storage"]], SCALE16 if c["source"] == "int16" else 1.0, c["zero_phase"])
    cube, w = state["cube"], state["weights"]
    if kind == "factors":
        return {"cf": postprocess.coherence_factor(cube, Dimension.receive, state["count"]),
                "pcf": postprocess.phase_coherence_factor(cube, w),
                "gcf": postprocess.generalized_coherence_factor(cube, c["m0"])}
    return postprocess.capon_minimum_variance(cube, w, c["nz"], c["nx"], c["l_elements"], c["k_samples"], 1.0 / 100,
                                              doForwardBackward=c["fb"])


def work(case):
    c = case
    size = {"fp32": 4, "fp16": 2, "bf16": 2}
    if c["kind"] == "demod":
        out = c["traces"] * (-(-c["l"] // c["decimation"]))
        taps = len(_taps(c))
        taps = 2 * taps - 1 if c["zero_phase"] else taps
        return {"bytes": c["traces"] * c["l"] * (2 if c["source"] == "int16" else 4) + out * 2 * size[c["storage"]],
                "flops": 4.0 * out * taps}
    if c["kind"] in ("factors", "capon"):
        p, f = c["nx"] * c["nz"], c["frames"]
        if c["kind"] == "factors":
            bins = 1 if c["m0"] <= 1 else 2 * c["m0"] + 1
            w = 4 * c["k"] * p if c["weights"] else 0
            return {"bytes": 8 * c["k"] * p * f + w + 40 * p * f, "flops": float(p * f * c["k"] * (8 + 60 + 8 * bins))}
        n, m = c["l_elements"], c["k"]
        rows = 2 * c["k_samples"] + 1
        return {"bytes": 8 * m * p * f + 4 * m * p + 8 * p * f,
                "flops": float(p * f * (rows * n * ((m - n + 1) + 2 * n) * 8 + 8 * n ** 3 / 3))}
    n, p = c["nx_el"] * c["ny_el"], c["nx"] * c["ny"] * c["nz"]
    el = 8 if c["complex"] else 4
    data = c["l"] * n * c["w"] * c["frames"]
    kept = {"both": 1, "transmit": n, "receive": c["w"], "none": n * c["w"]}[c["dim"]]
    if c["kind"] == "ensemble":
        moved = data * 4
    elif c["kind"] in ("table", "go"):
        moved = data * el + 8 * p * (n + c["w"])
    else:
        moved = data * size[c["storage"]] * (2 if c["complex"] else 1) + 12 * p
    # units with a receive weight: the aperture covers z / F-number of the array around the pixel
    scan, probe = _scan(c), _probe(c)
    xyz = torch.as_tensor(scan.xyz[(np.arange(512) * 0.6180339887 % 1.0 * p).astype(int)], dtype=torch.float64)
    active = float((_receive_apodization(c, torch.as_tensor(probe.xyz), xyz) != 0).double().mean())
    return {"bytes": moved + p * kept * c["frames"] * el + 24 * p * c["frames"] * c["epilogue"],
            "flops": (22.0 if c["complex"] else 10.0) * active * p * n * c["w"] * c["frames"]}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------

def _das64(c, x, tau_tx, rx_of, fd, phase):
    """Sum of a frame (W, N, L) over channels and / or waves: [Wk, Nk, P].
    ``rx_of(a, b)``: receive delays and weights [b - a, P] of channels a .. b."""
    W, N, L = x.shape
    P = tau_tx.shape[1]
    fs, t0 = 4 * c["f0"], c["t0"]
    dim = c["dim"]
    dt = torch.complex128 if x.is_complex() else torch.float64
    out = torch.zeros(W if dim == "receive" else 1, N if dim == "transmit" else 1, P, dtype=dt, device=x.device)
    turn = lambda tau: torch.polar(torch.ones_like(tau), 2 * math.pi * fd * tau) if x.is_complex() else 1.0  # noqa: E731
    step = max(1, (1 << 24) // P)
    for a in range(0, N, step):
        tau_rx, apo = rx_of(a, min(a + step, N))
        weight = apo * turn(tau_rx)
        for w in range(W):
            s = (tau_tx[w] + tau_rx - t0) * fs
            i = torch.floor(s)
            ok = (i > 0) & (i < L - 1)
            b = s - i
            i = i.clamp(0, L - 2).long()
            v = x[w, a:a + step]
            v = (v.gather(1, i) * (1 - b) + v.gather(1, i + 1) * b) * (weight * ok) * turn(tau_tx[w])
            if dim == "transmit":
                out[0, a:a + step] += v
            else:
                out[w if dim == "receive" else 0, 0] += v.sum(0)
    return out * phase if phase is not None else out


def _exact_das(c, seed):
    dev = torch.device("cuda", 0)
    scan = _scan(c)
    xyz, el = _t(scan.xyz, dev), _t(_probe(c).xyz, dev)
    tau_tx = _transmit_tau(c, xyz)
    ph = _pixel_phase(c, scan)
    ph = None if ph is None else torch.as_tensor(ph, device=dev)
    fd = _fd(c)
    if c["kind"] == "table":
        tau_tx, ph = tau_tx.float().double(), None

    def rx_of(a, b):
        tau, apo = _distance(el[a:b], xyz) / C, _receive_apodization(c, el[a:b], xyz)
        return (tau.float().double(), apo.float().double()) if c["kind"] == "table" else (tau, apo)

    if c["kind"] == "ensemble":
        x = _int16_iq(c, seed, dev)
    elif c["kind"] in ("table", "go"):
        x = _channels(c, seed, dev)
    else:
        x = _stored(c, _channels(c, seed, dev))
    frames = []
    for f in range(c["frames"]):
        v = x[f].double()
        if c["kind"] == "ensemble":
            v = torch.view_as_complex(v * SCALE16)
        elif c["kind"] in ("fast", "plan") and c["complex"]:
            v = torch.view_as_complex(v)
        elif c["kind"] in ("go", "table") and c["complex"]:
            v = x[f].to(torch.complex128)
        if c["kind"] == "go" and not c["complex"]:  # analytic signal along time
            L = c["l"]
            h = torch.zeros(L, dtype=torch.float64, device=dev)
            h[0] = 1.0
            h[1:(L + 1) // 2] = 2.0
            if L % 2 == 0:
                h[L // 2] = 1.0
            v = torch.fft.ifft(torch.fft.fft(v, dim=-1) * h, dim=-1)
        frames.append(_das64(c, v, tau_tx, rx_of, fd, ph))
    cube = torch.stack(frames)
    if c["kind"] == "go":
        return cube.permute(3, 2, 1, 0)
    if c["kind"] in ("table", "ensemble"):
        return cube
    out = {"cube": cube, "flags": None}
    if c["epilogue"]:
        y = cube[:, 0]  # (F, N, P)
        total = y.sum(1)
        m = (_receive_apodization(c, el, xyz) > 0.16).sum(0)
        cf = torch.nan_to_num(total.abs() ** 2 / (y.abs() ** 2).sum(1) / m, nan=0.0)
        re = y.real
        out.update(das=total, cf=cf, cf_image=cf * total,
                   sdmas=0.5 * ((re.sign() * re.abs().sqrt()).sum(1) ** 2 - re.abs().sum(1)))
    return out


def _exact_demod(c, seed):
    dev = torch.device("cuda", 0)
    rf, b, d = _rf(c, seed, dev), _taps(c).astype(np.float64), c["decimation"]
    n, L = len(b), c["l"]
    turn = torch.arange(L, device=dev, dtype=torch.float64) / c["over"]
    osc = torch.polar(torch.ones_like(turn), -2 * math.pi * (turn - turn.floor()))
    out = torch.empty(c["traces"], -(-L // d), 2, dtype=torch.float64, device=dev)

    def fir(x):  # causal, the input held at its first value before the trace
        x = torch.cat([x[:, :1].expand(-1, n - 1), x], 1)
        return sum(float(b[k]) * x[:, n - 1 - k:x.shape[1] - k] for k in range(n))

    for a in range(0, c["traces"], 4096):
        mix = rf[a:a + 4096].double() * (SCALE16 if c["source"] == "int16" else 1.0) * osc
        if c["zero_phase"]:  # filtfilt: odd extension by 3 n, steady-state starts
            e = 3 * n
            x = torch.cat([2 * mix[:, :1] - mix[:, 1:e + 1].flip(1), mix, 2 * mix[:, -1:] - mix[:, -e - 1:-1].flip(1)], 1)
            y = fir(fir(x).flip(1)).flip(1)[:, e:e + L]
        else:
            y = fir(torch.cat([torch.zeros_like(mix[:, :n]), mix], 1))[:, n:]
        out[a:a + 4096] = torch.view_as_real(y[:, ::d].contiguous())
    return out


def _exact_factors(c, seed):
    dev = torch.device("cuda", 0)
    cube = _cube(c, seed, dev)[:, 0].to(torch.complex128)  # (F, K, P)
    F, K, P = cube.shape
    weights = _cube_weights(c, dev) if c["weights"] else None
    total, energy = cube.sum(1), (cube.abs() ** 2).sum(1)
    m = (weights > 0.16).sum(0).double() if c["weights"] else float(K)
    cf = torch.nan_to_num(total.abs() ** 2 / energy / m, nan=0.0)
    w = weights.double()[None] if c["weights"] else torch.ones(1, K, P, dtype=torch.float64, device=dev)
    phi = cube.angle()

    def spread(v):  # weighted variance
        mean = (w * v).sum(1, keepdim=True) / w.sum(1, keepdim=True)
        return (w * (v - mean) ** 2).sum(1) / w.sum(1)

    psi = torch.where(phi <= 0, phi + math.pi, phi - math.pi)
    fca = (1 - torch.minimum(spread(phi).sqrt(), spread(psi).sqrt()) * math.sqrt(3) / math.pi).clamp(min=0)
    fca = torch.nan_to_num(fca, nan=0.0)
    fcc = 1 - (spread(phi.cos()) + spread(phi.sin())).sqrt()
    bins = torch.fft.fft(cube, dim=1).abs() ** 2
    low = bins[:, :1].sum(1)
    if c["m0"] > 1:
        low = bins[:, :c["m0"] + 1].sum(1) + bins[:, K - c["m0"]:].sum(1)
    gcf = torch.nan_to_num(low / (K * energy), nan=0.0)
    shape = lambda v: v.reshape(F, 1, 1, P)  # noqa: E731
    return {"cf": {"CF": shape(cf), "image": shape(cf * total)}, "pcf": {"FCA": fca, "FCC": fcc, "image": fcc * total},
            "gcf": {"GCF": gcf, "image": gcf * total}}


def _exact_capon(c, seed):
    dev = torch.device("cuda", 0)
    cube = _cube(c, seed, dev)[:, 0].to(torch.complex128)  # (F, M, P)
    F, M, P = cube.shape
    nz, nx, K = c["nz"], c["nx"], c["k_samples"]
    active = _cube_weights(c, dev).abs() > 0.16
    index = torch.arange(M, device=dev)[:, None]
    count = active.sum(0)
    first = torch.where(active, index, M).amin(0)
    last = torch.where(active, index, -1).amax(0)
    sides, which = torch.unique(torch.stack([first, last, count]), dim=1, return_inverse=True)
    out = torch.empty(F, P, dtype=torch.complex128, device=dev)
    for f in range(F):
        x = cube[f].t().reshape(nx, nz, M)
        pad = torch.zeros(nx, K, M, dtype=x.dtype, device=dev)
        rows = torch.cat([pad, x, pad], 1).unfold(1, 2 * K + 1, 1).reshape(P, M, 2 * K + 1)  # zero rows add nothing
        for j in range(sides.shape[1]):
            a, b, n = (int(v) for v in sides[:, j])
            pixels = (which == j).nonzero()[:, 0]
            L = max(1, min(int(np.floor(np.float32(c["l_elements"]) / np.float32(M) * np.float32(n))), n - 1)) if n > 1 else 0
            if n < 2 or b - L + 1 < a:
                out[f, pixels] = x.reshape(P, M)[pixels].sum(1)
                continue
            for p in pixels.split(2048):
                sub = rows[p][:, a:b + 1].permute(0, 2, 1).unfold(2, L, 1).reshape(p.numel(), -1, L)
                R = sub.conj().transpose(1, 2) @ sub / ((2 * K + 1) * (n - L + 1))
                if c["fb"]:
                    R = 0.5 * (R + R.conj().flip(1, 2))
                load = R.diagonal(dim1=1, dim2=2).real.sum(1) / L / 100
                R = R + load[:, None, None] * torch.eye(L, dtype=R.dtype, device=dev)
                v = torch.linalg.solve(R, torch.ones(p.numel(), L, 1, dtype=R.dtype, device=dev))[:, :, 0]
                v = v / v.sum(1, keepdim=True)
                own = x.reshape(P, M)[p][:, a:b + 1].unfold(1, L, 1).sum(1)
                out[f, p] = (v * own).sum(1).conj() * (n / (n - L + 1))
    return out


def exact(case, seed):
    if case["kind"] == "demod":
        return _exact_demod(case, seed)
    if case["kind"] == "factors":
        return _exact_factors(case, seed)
    if case["kind"] == "capon":
        return _exact_capon(case, seed)
    return _exact_das(case, seed)
