"""The fast kernels at the edges of their stages and windows, against the FP64 oracle.

Stages hold 8 x 4, 16 x 2 or 2 x 16 (channel, wave) slots of 80 or 160 samples: channel
and wave counts around multiples of those, coarse pixel grids whose windows need the
longer slots, traces that end inside the windows, odd real traces, and several frames of
one persistent work item.  The bar is the FP32-storage bar of the fast path against the
oracle, 2e-4 (sample positions and phases in FP32)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import fast, geometry
from ustb_gb300.enums import Precision, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan, Point, Probe, Wave

pytestmark = pytest.mark.gpu

BAR = 2e-4
C, FS, F0, T0 = 1540.0, 20e6, 5e6, 2e-6


def setup(N, W, L, F, cplx, pitch_px, seed=0, diverging=False):
    rng = np.random.default_rng(seed)
    probe = Probe.linear_array(N, 0.3e-3)
    ang = np.deg2rad(np.linspace(-12, 12, W)) if W > 1 else np.zeros(1)
    seq = [Wave(source=Point(-10e-3, float(a), 0.0)) if diverging else Wave.plane(float(a)) for a in ang]
    scan = LinearScan(np.arange(-15, 16) * pitch_px, 8e-3 + np.arange(37) * pitch_px)
    x = rng.standard_normal((L + 4, N, W, F)) + (1j * rng.standard_normal((L + 4, N, W, F)) if cplx else 0)
    x = sum(k * x[i:i + L] for i, k in enumerate((1, 4, 6, 4, 1))) / 16  # band-limited
    return probe, seq, scan, x.astype(np.complex64 if cplx else np.float32)


def oracle(probe, seq, scan, x, dim, rx, fd):
    tabs = (Apodization().wave_apodization(seq, scan), rx.aperture_apodization(probe, scan),
            geometry.transmit_delay(seq, scan), geometry.receive_delay(probe, scan, C))
    return O.das_f64(x.astype(np.complex128), FS, T0, *tabs, fd, dim)


def tensors(probe, seq, scan, x, rx, shape, dev):
    fd = F0 if np.iscomplexobj(x) else 0.0
    g = fast.FastGeometry(probe, scan, seq, FS, T0, fd, C, dev, rx, None, stage_shape=shape)
    ch = torch.from_numpy(np.ascontiguousarray(x.transpose(3, 2, 1, 0))).to(dev)
    return g, fast.convert_channels(ch, Precision.fp32), fd


def rel(got, want):
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


@pytest.mark.parametrize("pitch_px", [0.1e-3, 0.16e-3])  # short and long sample windows
@pytest.mark.parametrize("shape, dim", [(1, 3), (2, 3), (3, 3), (1, 1), (2, 2), (3, 2), (2, 0)])
@pytest.mark.parametrize("N, W", [(7, 1), (16, 2), (17, 5), (33, 17)])
def test_stage_remainders(cuda_dev, N, W, shape, dim, pitch_px):
    probe, seq, scan, x = setup(N, W, 512, 1, True, pitch_px, seed=N + W)
    rx = Apodization(window=Window.tukey25, f_number=1.2)
    g, st, fd = tensors(probe, seq, scan, x, rx, shape, cuda_dev)
    out = fast.das_fast(st, Precision.fp32, True, g, dim, L=512)["cube"].cpu().numpy().transpose(3, 2, 1, 0)
    assert rel(out, oracle(probe, seq, scan, x, dim, rx, fd)) <= BAR


@pytest.mark.parametrize("L", [330, 331])  # even and odd traces that end inside the deepest windows
@pytest.mark.parametrize("shape", [1, 2, 3])
@pytest.mark.parametrize("W, diverging", [(1, False), (6, True)])
def test_real_traces_and_their_ends(cuda_dev, W, diverging, shape, L):
    probe, seq, scan, x = setup(19, W, L, 1, False, 0.2e-3, seed=L, diverging=diverging)
    rx = Apodization(window=Window.tukey50, f_number=0.8)
    g, st, fd = tensors(probe, seq, scan, x, rx, shape, cuda_dev)
    out = fast.das_fast(st, Precision.fp32, False, g, 3, L=L)["cube"].cpu().numpy().transpose(3, 2, 1, 0)
    assert rel(out, oracle(probe, seq, scan, x.astype(np.complex64), 3, rx, 0.0).real) <= BAR


@pytest.mark.parametrize("dim, shape", [(3, 1), (3, 2), (2, 2), (1, 1)])
@pytest.mark.parametrize("F", [2, 11])
def test_frames_of_one_persistent_item(cuda_dev, F, dim, shape):
    probe, seq, scan, x = setup(18, 3, 420, F, True, 0.12e-3, seed=F)
    rx = Apodization(window=Window.hanning, f_number=1.0)
    g, st, fd = tensors(probe, seq, scan, x, rx, shape, cuda_dev)
    r = fast.Request(st, Precision.fp32, True, g, dim, F=F, L=420)
    fast.das_fast_batch([r], max_ctas=1)  # one pair of CTAs: every item takes several frames
    out = r.outputs["cube"].cpu().numpy().transpose(3, 2, 1, 0)
    assert rel(out, oracle(probe, seq, scan, x, dim, rx, fd)) <= BAR
