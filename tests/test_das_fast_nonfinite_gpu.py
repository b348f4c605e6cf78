"""Pixel positions that are not numbers, on the fast path."""
import numpy as np
import pytest
import torch

from ustb_gb300 import fast
from ustb_gb300.enums import Precision, Wavefront, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan, Probe, Wave

pytestmark = pytest.mark.gpu

C, FS, F0, T0, L = 1540.0, 20e6, 5e6, 2e-6, 400
SCAN = LinearScan(np.linspace(-3e-3, 3e-3, 31), np.linspace(6e-3, 11e-3, 43))


@pytest.mark.parametrize("wave", [Wave.plane(0.0), Wave(Wavefront.photoacoustic)])
@pytest.mark.parametrize("axis", [0, 1])
def test_pixel_without_a_position(cuda_dev, axis, wave):
    """A pixel whose lateral position is NaN has no receive weight (das_c's windows are 0 at
    a NaN ratio): 0; its neighbours are as without it."""
    rng = np.random.default_rng(axis)
    N, bad = 17, 200
    ch = torch.from_numpy(rng.standard_normal((1, 1, N, L)).astype(np.float32)).to(cuda_dev)
    rx = Apodization(window=Window.tukey25, f_number=1.2)
    outs = []
    for broken in (False, True):
        g = fast.FastGeometry(Probe.linear_array(N, 0.3e-3), SCAN, [wave], FS, T0, 0.0, C, cuda_dev, rx, None)
        if broken:
            g.d_px.view(-1, 3)[bad, axis] = float("nan")
        outs.append(fast.das_fast(ch, Precision.fp32, False, g, 3, L=L)["cube"].flatten())
    assert outs[1][bad] == 0 and outs[0][bad] != 0
    keep = torch.arange(SCAN.N_pixels, device=cuda_dev) != bad
    assert torch.linalg.vector_norm((outs[1] - outs[0])[keep]) <= 1e-6 * torch.linalg.vector_norm(outs[0])
