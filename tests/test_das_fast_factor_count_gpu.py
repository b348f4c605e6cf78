"""The number of channels that the fused coherence factor divides by."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import fast
from ustb_gb300.enums import Precision, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan, Probe, Wave

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stage_shape", [0, 3])
@pytest.mark.parametrize("N", [1, 9, 16, 23])
@pytest.mark.parametrize("threshold", [-1.0, 0.16])
def test_channels_past_the_last_are_not_counted(cuda_dev, N, threshold, stage_shape):
    """Every channel's weight exceeds the threshold: M = N, also where N does not fill its
    last group of channels and the threshold is below 0 (the bar: FP32 sums, 1e-5)."""
    rng = np.random.default_rng(N)
    L = 300
    scan = LinearScan(np.linspace(-2e-3, 2e-3, 20), np.linspace(5e-3, 7e-3, 30))
    rx = Apodization(window=Window.boxcar, f_number=0.1)
    g = fast.FastGeometry(Probe.linear_array(N, 0.3e-3), scan, [Wave.plane(0.0)], 20e6, 1e-6, 5e6, 1540.0, cuda_dev, rx,
                          None, cf_threshold=threshold, stage_shape=stage_shape)
    ch = torch.from_numpy(rng.standard_normal((1, 1, N, L, 2)).astype(np.float32)).to(cuda_dev)
    out = fast.das_fast(ch, Precision.fp32, True, g, 2, L=L, epilogue=True)
    kept = out["cube"][0, 0].cpu().numpy().T  # [P, N]
    want, _ = O.coherence_factor(kept, np.full(scan.N_pixels, N))
    got = out["cf"][0].cpu().numpy()
    assert np.linalg.norm(got - want[:, 0]) <= 1e-5 * np.linalg.norm(want)
