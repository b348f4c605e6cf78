"""Requests whose tables leave room for one CTA on an SM (a whole tile each), around the
number of channels and waves where that begins, against the FP64 oracle.  The bar is the
FP32-storage bar of the fast path, 2e-4; 16-bit samples are compared as they are stored."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import fast, geometry
from ustb_gb300.enums import Precision, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan3D, Probe, Wave

pytestmark = pytest.mark.gpu

C, FS, F0, T0, L = 1540.0, 20e6, 5e6, 2e-6, 460


def case(nx, ny, W, F, cplx, storage, dev, **kw):
    rng = np.random.default_rng(nx * ny + W)
    probe = Probe.matrix_array(nx, ny, 0.2e-3)
    N = nx * ny
    seq = [Wave.plane(float(a)) for a in np.deg2rad(np.linspace(-6, 6, W))]
    scan = LinearScan3D(np.linspace(-3e-3, 3e-3, 9), np.linspace(6e-3, 12e-3, 31), np.linspace(-1e-3, 1e-3, 5))
    rx = Apodization(window=Window.tukey25, f_number=0.9)
    fd = F0 if cplx else 0.0
    g = fast.FastGeometry(probe, scan, seq, FS, T0, fd, C, dev, rx, None, **kw)
    x = torch.from_numpy(rng.standard_normal((F, W, N, L) + ((2,) if cplx else ())).astype(np.float32)).to(dev)
    x = (x[..., :-2, :] + 2 * x[..., 1:-1, :] + x[..., 2:, :]) / 4 if cplx else (x[..., :-2] + 2 * x[..., 1:-1] + x[..., 2:]) / 4
    st = x.contiguous().to(fast.TORCH_STORE[storage])
    v = st.float().cpu().numpy().astype(np.float64)
    v = (v[..., 0] + 1j * v[..., 1] if cplx else v).astype(np.complex128).transpose(3, 2, 1, 0)
    tabs = (Apodization().wave_apodization(seq, scan), rx.aperture_apodization(probe, scan),
            geometry.transmit_delay(seq, scan), geometry.receive_delay(probe, scan, C))
    return g, st, lambda dim: O.das_f64(v, FS, T0, *tabs, fd, dim)


@pytest.mark.parametrize("nx, ny, W, F, cplx, storage", [
    (34, 34, 1, 1, True, Precision.fp32), (35, 34, 1, 2, True, Precision.fp16), (35, 35, 3, 1, True, Precision.fp32),
    (16, 16, 300, 1, True, Precision.bf16), (40, 40, 2, 2, False, Precision.fp32), (8, 8, 700, 1, False, Precision.fp32)])
@pytest.mark.parametrize("dim", [3, 2, 1])
def test_against_the_oracle(cuda_dev, nx, ny, W, F, cplx, storage, dim):
    g, st, want = case(nx, ny, W, F, cplx, storage, cuda_dev)
    want = want(dim) if cplx else want(dim).real
    out = fast.das_fast(st, storage, cplx, g, dim, F=F, L=L - 2)["cube"]
    r = fast.Request(st, storage, cplx, g, dim, F=F, L=L - 2)
    fast.das_fast_batch([r], max_ctas=7)
    for y in (out, r.outputs["cube"]):
        y = y.cpu().numpy().transpose(3, 2, 1, 0)
        assert np.linalg.norm(y - want) <= 2e-4 * np.linalg.norm(want)


@pytest.mark.parametrize("parts", [1, 3])
def test_parts_asked_for(cuda_dev, parts):
    g, st, want = case(36, 35, 5, 1, True, Precision.fp32, cuda_dev, ctas_per_tile=parts)
    out = fast.das_fast(st, Precision.fp32, True, g, 3, L=L - 2)["cube"].cpu().numpy().transpose(3, 2, 1, 0)
    want = want(3)
    assert np.linalg.norm(out - want) <= 2e-4 * np.linalg.norm(want)


def test_one_launch_beside_few_channels(cuda_dev):
    made = [case(n, n, 3, 1, True, Precision.fp16, cuda_dev) for n in (35, 9)]
    reqs = [fast.Request(st, Precision.fp16, True, g, 3, L=L - 2) for g, st, _ in made]
    scratch = fast.das_fast_batch(reqs, max_ctas=9)  # (bounded: persistent)
    assert int((scratch[1:] != 0).sum()) == 1
    for r, (_, _, want) in zip(reqs, made):
        w = want(3)
        assert np.linalg.norm(r.outputs["cube"].cpu().numpy().transpose(3, 2, 1, 0) - w) <= 2e-4 * np.linalg.norm(w)
