"""Sub-tiles whose work several CTAs share, against the FP64 oracle: parts of the stages
with their sums added by the last part (dimension.both), parts of the channel groups or
wave chunks (transmit, receive), whole groups without a weight between and at the ends,
more parts than stages, and the same bits on every run.  The bar is the FP32-storage bar
of the fast path against the oracle, 2e-4."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import fast, geometry
from ustb_gb300.enums import Precision, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan, Probe, Wave

pytestmark = pytest.mark.gpu

BAR = 2e-4
C, FS, F0, T0, L = 1540.0, 20e6, 5e6, 2e-6, 640


def case(N, W, F, cplx, f_number, dev, seed, **kw):
    rng = np.random.default_rng(seed)
    probe = Probe.linear_array(N, 0.3e-3)
    seq = [Wave.plane(float(a)) for a in np.deg2rad(np.linspace(-9, 9, W) if W > 1 else np.zeros(1))]
    scan = LinearScan(np.linspace(-6e-3, 6e-3, 41), np.linspace(6e-3, 16e-3, 61))
    x = rng.standard_normal((L + 4, N, W, F)) + (1j * rng.standard_normal((L + 4, N, W, F)) if cplx else 0)
    x = sum(k * x[i:i + L] for i, k in enumerate((1, 4, 6, 4, 1))) / 16  # band-limited
    x = x.astype(np.complex64 if cplx else np.float32)
    rx = Apodization(window=Window.tukey25, f_number=f_number)
    fd = F0 if cplx else 0.0
    g = fast.FastGeometry(probe, scan, seq, FS, T0, fd, C, dev, rx, None, **kw)
    st = fast.convert_channels(torch.from_numpy(np.ascontiguousarray(x.transpose(3, 2, 1, 0))).to(dev), Precision.fp32)
    tabs = (Apodization().wave_apodization(seq, scan), rx.aperture_apodization(probe, scan),
            geometry.transmit_delay(seq, scan), geometry.receive_delay(probe, scan, C))
    want = lambda dim: O.das_f64(x.astype(np.complex128), FS, T0, *tabs, fd, dim)
    return g, st, want


def rel(got, want):
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


@pytest.mark.parametrize("dim, cplx", [(3, True), (3, False), (2, True), (2, False), (1, True), (1, False)])
@pytest.mark.parametrize("N, W, F", [(1, 1, 1), (9, 33, 1), (130, 5, 2), (65, 50, 1)])
def test_parts(cuda_dev, N, W, F, dim, cplx):
    g, st, want = case(N, W, F, cplx, 3.0, cuda_dev, N + W)
    run = lambda: fast.das_fast(st, Precision.fp32, cplx, g, dim, F=F, L=L)["cube"]
    out = run()
    want = want(dim)
    assert rel(out.cpu().numpy().transpose(3, 2, 1, 0), want if cplx else want.real) <= BAR
    assert all(torch.equal(out, run()) for _ in range(3))


@pytest.mark.parametrize("parts", [1, 2, 3, 4])
def test_parts_asked_for(cuda_dev, parts):
    g, st, want = case(37, 7, 2, True, 1.5, cuda_dev, parts, ctas_per_tile=parts)
    run = lambda: fast.das_fast(st, Precision.fp32, True, g, 3, F=2, L=L)["cube"]
    out = run()
    assert rel(out.cpu().numpy().transpose(3, 2, 1, 0), want(3)) <= BAR
    assert torch.equal(out, run())


@pytest.mark.parametrize("N, W, F", [(3, 1, 1), (65, 7, 1), (130, 2, 2)])
def test_parts_of_the_epilogue(cuda_dev, N, W, F):
    """The epilogue's sums over channels in parts, against the persistent launch, which sums
    all channels in one CTA: 130 terms in another order differ by under 1e-6 of the sums;
    the factors and DMAS square and divide them: 1e-5."""
    g, st, _ = case(N, W, F, True, 2.0, cuda_dev, N * W)
    run = lambda: fast.das_fast(st, Precision.fp32, True, g, 2, F=F, L=L, epilogue=True)
    got, again = run(), run()
    r = fast.Request(st, Precision.fp32, True, g, 2, F=F, L=L, epilogue=True)
    fast.das_fast_batch([r])
    for k, want in r.outputs.items():
        v = got[k]
        assert torch.equal(v, again[k])
        ok = torch.isfinite(want.abs())  # a factor is infinite where no weight exceeds the threshold
        assert torch.equal(v[~ok], want[~ok])
        assert torch.linalg.vector_norm((v - want)[ok]) <= 1e-5 * torch.linalg.vector_norm(want[ok]), k
