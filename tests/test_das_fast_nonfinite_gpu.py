"""Samples and pixel positions that are not finite, on the fast path: they reach the pixels
that das_c's formula gives them, and no others."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import fast, geometry
from ustb_gb300.enums import Precision, Wavefront, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan, Probe, Wave

pytestmark = pytest.mark.gpu

C, FS, F0, T0, L = 1540.0, 20e6, 5e6, 2e-6, 400
SCAN = LinearScan(np.linspace(-3e-3, 3e-3, 31), np.linspace(6e-3, 11e-3, 43))


def sequence(W):
    return [Wave.plane(float(a)) for a in np.deg2rad(np.linspace(-9, 9, W))]


@pytest.mark.parametrize("storage", [Precision.fp32, Precision.fp16])
@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("dim, shape", [(3, 0), (3, 1), (3, 2), (3, 3), (2, 0), (2, 3), (1, 0), (1, 1)])
@pytest.mark.parametrize("W, silent", [(3, ()), (11, ()), (15, ()), (12, (9,)), (19, (0, 6, 18))])
def test_bad_samples_stay_where_they_are_read(cuda_dev, W, silent, dim, shape, cplx, storage):
    """Windows of waves with an infinite and a NaN sample are left in the stage buffers;
    padding waves and waves without a weight, whose places they hold, add nothing."""
    rng = np.random.default_rng(W)
    N = 33
    probe, seq = Probe.linear_array(N, 0.3e-3), sequence(W)
    weights = np.ones(W)
    weights[list(silent)] = 0.0
    rx, tx = Apodization(), Apodization(apodization_vector=weights)
    x = rng.standard_normal((1, W, N, L)) + (1j * rng.standard_normal((1, W, N, L)) if cplx else 0)
    x[0, 1::2, 20, 150] = np.nan
    x[0, 3::4, 9, 170] = np.inf
    fd = F0 if cplx else 0.0
    g = fast.FastGeometry(probe, SCAN, seq, FS, T0, fd, C, cuda_dev, rx, tx, stage_shape=shape)
    ch = torch.from_numpy(x.astype(np.complex64 if cplx else np.float32)).to(cuda_dev)
    out = fast.das_fast(fast.convert_channels(ch, storage), storage, cplx, g, dim, L=L)["cube"].cpu().numpy()
    r = fast.Request(fast.convert_channels(ch, storage), storage, cplx, g, dim, L=L)
    fast.das_fast_batch([r])
    # what das_c reads: samples floor(s) and floor(s) + 1 of every wave with a weight
    tau_tx, tau_rx = geometry.transmit_delay(seq, SCAN), geometry.receive_delay(probe, SCAN, C)  # [P, W], [P, N]
    s = (tau_tx[:, :, None] + tau_rx[:, None, :] - T0) * FS
    i = np.floor(s).astype(int)
    tie = np.zeros((SCAN.N_pixels, W, N), bool)  # FP32 positions may fall on the other side
    hit = np.zeros_like(tie)
    for n, j, first, step in ((20, 150, 1, 2), (9, 170, 3, 4)):
        for w in range(first, W, step):
            if weights[w]:
                hit[:, w, n] = (i[:, w, n] == j) | (i[:, w, n] == j - 1)
                tie[:, w, n] = np.abs(s[:, w, n] - np.array([j - 1, j, j + 1])[:, None]).min(0) < 2e-3
    over = {3: (1, 2), 2: (1,), 1: (2,)}[dim]
    hit, tie = hit.any(over, keepdims=True), tie.any(over, keepdims=True)
    want = np.moveaxis(~hit, 0, -1)  # [W, N, P] as the output's
    sure = np.moveaxis(~tie, 0, -1)
    assert hit.any() and want.any()
    for y in (out, r.outputs["cube"].cpu().numpy()):
        assert np.array_equal(np.isfinite(y[0])[sure], want[sure])


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
