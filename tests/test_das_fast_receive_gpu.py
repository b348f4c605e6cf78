"""dimension.receive at the remainders of its stage shapes (16 channels x 2 waves up to
two waves, 8 x 4 up to eight, 4 x 8 beyond), several frames, grid and persistent
launches, against the 2 x 16 stages that a geometry can ask for.  Both form each unit
alike and add a wave's channels in order; 1e-6 leaves room for another order."""
import numpy as np
import pytest
import torch

from ustb_gb300 import fast
from ustb_gb300.enums import Precision, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan, Probe, Wave

pytestmark = pytest.mark.gpu

C, FS, F0, T0, L = 1540.0, 20e6, 5e6, 2e-6, 512


@pytest.mark.parametrize("pitch_px", [0.08e-3, 0.2e-3])  # short and long sample windows
@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("N, W", [(1, 1), (17, 1), (33, 2), (15, 3), (9, 4), (25, 5), (8, 17), (5, 9)])
def test_receive_images(cuda_dev, N, W, cplx, pitch_px):
    rng = np.random.default_rng(N * 32 + W)
    probe = Probe.linear_array(N, 0.3e-3)
    seq = [Wave.plane(float(a)) for a in np.deg2rad(np.linspace(-9, 9, W) if W > 1 else np.zeros(1))]
    scan = LinearScan(np.arange(-14, 15) * pitch_px, 7e-3 + np.arange(39) * pitch_px)
    x = rng.standard_normal((L + 4, N, W, 2)) + (1j * rng.standard_normal((L + 4, N, W, 2)) if cplx else 0)
    x = sum(k * x[i:i + L] for i, k in enumerate((1, 4, 6, 4, 1))) / 16  # band-limited
    x = x.astype(np.complex64 if cplx else np.float32)
    rx = Apodization(window=Window.hamming, f_number=1.4)
    fd = F0 if cplx else 0.0
    st = fast.convert_channels(torch.from_numpy(np.ascontiguousarray(x.transpose(3, 2, 1, 0))).to(cuda_dev), Precision.fp32)
    g, general = (fast.FastGeometry(probe, scan, seq, FS, T0, fd, C, cuda_dev, rx, None, stage_shape=s) for s in (0, 1))
    want = fast.das_fast(st, Precision.fp32, cplx, general, 1, F=2, L=L)["cube"]
    out = fast.das_fast(st, Precision.fp32, cplx, g, 1, F=2, L=L)["cube"]
    r = fast.Request(st, Precision.fp32, cplx, g, 1, F=2, L=L)
    fast.das_fast_batch([r])
    for y in (out, r.outputs["cube"]):
        assert torch.linalg.vector_norm(y - want) <= 1e-6 * torch.linalg.vector_norm(want)
