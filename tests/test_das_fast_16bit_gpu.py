"""Complex FP16 and bfloat16 channel data: entries kept in the storage type (the library's
own stage shapes) against FP32 entries (a shape that is asked for).  Both form a unit's
values and sum them alike; 1e-6 leaves room for another order.  Traces that end inside the
windows, odd lengths, short and long windows, infinities and NaN in samples that no
pixel reaches and in some that pixels do."""
import numpy as np
import pytest
import torch

from ustb_gb300 import fast
from ustb_gb300.enums import Precision, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan, Probe, Wave

pytestmark = pytest.mark.gpu

C, FS, F0, T0 = 1540.0, 20e6, 5e6, 2e-6


@pytest.mark.parametrize("precision", [Precision.fp16, Precision.bf16])
@pytest.mark.parametrize("dim, shape", [(3, 3), (2, 3), (1, 1)])
@pytest.mark.parametrize("N, W, L, pitch_px", [(1, 1, 330, 0.1e-3), (17, 2, 331, 0.1e-3), (9, 5, 512, 0.2e-3), (20, 11, 513, 0.06e-3)])
def test_stored_entries(cuda_dev, N, W, L, pitch_px, dim, shape, precision):
    rng = np.random.default_rng(N + W + L)
    probe = Probe.linear_array(N, 0.3e-3)
    seq = [Wave.plane(float(a)) for a in np.deg2rad(np.linspace(-9, 9, W) if W > 1 else np.zeros(1))]
    scan = LinearScan(np.arange(-14, 15) * pitch_px, 7e-3 + np.arange(41) * pitch_px)
    rx = Apodization(window=Window.tukey25, f_number=1.4)
    ch = torch.from_numpy(rng.standard_normal((2, W, N, L, 2)).astype(np.float32)).to(cuda_dev)
    ch[1, :, 0, 5] = float("inf")  # before the image's first samples
    ch[1, 0, N // 2, 200] = float("nan")
    st = ch.to(torch.float16 if precision == Precision.fp16 else torch.bfloat16)
    outs = []
    for s in (0, shape):
        g = fast.FastGeometry(probe, scan, seq, FS, T0, F0, C, cuda_dev, rx, None, stage_shape=s)
        outs.append(fast.das_fast(st, precision, True, g, dim, F=2, L=L)["cube"])
        r = fast.Request(st, precision, True, g, dim, F=2, L=L)
        fast.das_fast_batch([r])
        outs.append(r.outputs["cube"])
    want = outs[2]
    ok = torch.isfinite(torch.view_as_real(want)).all(-1)
    assert ok.any()
    for y in outs:
        assert torch.equal(torch.isfinite(torch.view_as_real(y)).all(-1), ok)
        assert torch.linalg.vector_norm((y - want)[ok]) <= 1e-6 * torch.linalg.vector_norm(want[ok])
