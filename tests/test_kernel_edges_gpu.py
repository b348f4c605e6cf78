"""Demodulation, coherence and Capon kernels at the edges of their splits, against the
FP64 oracles: remainders of the output, tap, trace and channel blocks, the smallest and
largest counts they take, unaligned input.  Bars are those of the kernels' other tests."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import postprocess, preprocess
from ustb_gb300.enums import Precision

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def iq(t):
    a = t.float().cpu().numpy()
    return a[..., 0] + 1j * a[..., 1]


@pytest.mark.parametrize("D, L, traces", [(1, 1, 3), (1, 9, 300), (2, 16, 1), (2, 1537, 7), (3, 500, 11), (5, 6001, 2),
                                          (7, 40, 40), (64, 3000, 3), (1, 2049, 2)])
@pytest.mark.parametrize("ntaps", [1, 4, 30, 257])
def test_causal_demodulation(cuda_dev, D, L, traces, ntaps):
    rng = np.random.default_rng(L + ntaps)
    fs, t0, fc = 20e6, 0.3e-6, 4.1e6
    rf = rng.standard_normal((traces, L)).astype(np.float32)
    taps = (rng.standard_normal(ntaps) / ntaps).astype(np.float32)
    got = preprocess.demodulate(torch.from_numpy(rf).to(cuda_dev), fs, t0, fc, taps, D, Precision.fp32, 0.5)
    want = O.fast_demodulation_f64(rf.T.astype(np.float64) * 0.5, fs, t0, fc, taps, D)
    assert rel(iq(got), want.T) <= 1e-5


@pytest.mark.parametrize("D, L, traces", [(1, 301, 5), (2, 2500, 3), (3, 305, 300), (6, 4001, 2)])
@pytest.mark.parametrize("ntaps", [1, 2, 33, 100])
def test_zero_phase_demodulation(cuda_dev, D, L, traces, ntaps):
    rng = np.random.default_rng(L * 3 + ntaps)
    fs, t0, fc = 20e6, 0.3e-6, 4.1e6
    rf = rng.standard_normal((traces, L)).astype(np.float32)
    taps = np.hamming(ntaps + 2)[1:-1]
    taps = (taps / taps.sum()).astype(np.float32)
    got = preprocess.demodulate(torch.from_numpy(rf).to(cuda_dev), fs, t0, fc, taps, D, Precision.fp32, 0.5,
                                zero_phase=True)
    want = O.zero_phase_demodulation_f64(rf.T.astype(np.float64) * 0.5, fs, t0, fc, taps, D)
    assert rel(iq(got), want.T) <= 1e-5


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("dtype", [np.int16, np.float32, np.float16])
def test_demodulation_of_rf_at_any_address(cuda_dev, dtype, shift):
    """A view that starts ``shift`` samples into its storage."""
    rng = np.random.default_rng(shift)
    rf = np.round(rng.standard_normal((6, 403)) * 300).astype(dtype)
    flat = torch.zeros(rf.size + shift, dtype=torch.from_numpy(rf).dtype, device=cuda_dev)
    flat[shift:] = torch.from_numpy(rf).reshape(-1).to(cuda_dev)
    taps = preprocess.lowpass_taps(5e6, 20e6).astype(np.float32)
    got = preprocess.demodulate(flat[shift:].view(6, 403), 20e6, 0.0, 5e6, taps, 2)
    want = O.fast_demodulation_f64(rf.T.astype(np.float64), 20e6, 0.0, 5e6, taps, 2)
    assert rel(iq(got), want.T) <= 1e-5


def cube_of(rng, P, K, F=1):
    c = rng.standard_normal((F, K, P)) + 1j * rng.standard_normal((F, K, P)) + 1.5 * rng.standard_normal((F, 1, P))
    c[:, :, 0] = 0  # a silent pixel
    return c.astype(np.complex64)


@pytest.mark.parametrize("K", [2, 3, 7, 64, 130, 1024])
@pytest.mark.parametrize("P, F", [(65, 2), (300, 1)])
def test_phase_coherence_counts(cuda_dev, K, P, F):
    rng = np.random.default_rng(K + P)
    c = cube_of(rng, P, K, F)
    w = rng.uniform(0, 1, (K, P)).astype(np.float32)
    w[rng.random((K, P)) < 0.3] = 0
    w[0] = 0.5  # every pixel keeps a weight
    got = postprocess.phase_coherence_factor(torch.from_numpy(c[:, None]).to(cuda_dev), torch.from_numpy(w).to(cuda_dev))
    for f in range(F):
        fca, fcc, img = O.phase_coherence_factor_f64(c[f].T, w.T)
        assert np.max(np.abs(got["FCA"][f].cpu().numpy() - fca)) <= 1e-4
        assert np.max(np.abs(got["FCC"][f].cpu().numpy() - fcc)) <= 1e-4
        assert rel(got["image"][f].cpu().numpy(), img) <= 1e-4


def test_phase_coherence_of_agreeing_and_extreme_values(cuda_dev):
    """Phases that agree closely (at any angle), and magnitudes whose squares leave FP32."""
    rng = np.random.default_rng(1)
    K, P = 48, 130
    ang = np.linspace(-np.pi, np.pi, P)[None, :] + 1e-3 * rng.standard_normal((K, P))
    mag = 10.0 ** rng.uniform(-25, 25, (1, P))
    c = (mag * np.exp(1j * ang)).astype(np.complex64)
    got = postprocess.phase_coherence_factor(torch.from_numpy(c[None, None]).to(cuda_dev))
    fca, fcc, _ = O.phase_coherence_factor_f64(c.T)
    assert np.max(np.abs(got["FCA"][0].cpu().numpy() - fca)) <= 1e-4
    assert np.max(np.abs(got["FCC"][0].cpu().numpy() - fcc)) <= 1e-4


@pytest.mark.parametrize("M0, K", [(0, 2), (1, 5), (2, 3), (3, 4), (4, 5), (4, 64), (5, 11), (6, 7), (7, 8), (7, 1024)])
def test_generalized_coherence_counts(cuda_dev, M0, K):
    rng = np.random.default_rng(M0 * 100 + K)
    c = cube_of(rng, 131, K, 2)
    got = postprocess.generalized_coherence_factor(torch.from_numpy(c[:, None]).to(cuda_dev), M0)
    for f in range(2):
        g, img = O.generalized_coherence_factor_f64(c[f].T, M0)
        assert np.max(np.abs(got["GCF"][f].cpu().numpy() - g)) <= 1e-5
        assert rel(got["image"][f].cpu().numpy(), img) <= 1e-5


@pytest.mark.parametrize("M, L, K", [(2, 1, 0), (9, 4, 2), (40, 32, 1), (64, 32, 5), (73, 20, 0), (130, 32, 9), (256, 32, 1)])
@pytest.mark.parametrize("fb", [False, True])
def test_capon_channel_counts(cuda_dev, M, L, K, fb):
    rng = np.random.default_rng(M + K)
    nz, nx = 9, 2
    d = 0.3 * (rng.standard_normal((nz, nx, M)) + 1j * rng.standard_normal((nz, nx, M)))
    d += np.exp(1j * 0.3 * np.arange(M)) * rng.standard_normal((nz, nx, 1))
    ap = np.ones((nz, nx, M))
    for iz in range(nz):  # apertures that start and end anywhere in the tiles
        ap[iz, :, :min(iz, M - 2)] = 0
        ap[iz, 1, M - min(2 * iz, (M - 2) // 2):] = 0
    cube = torch.from_numpy(np.ascontiguousarray(d.transpose(2, 1, 0).reshape(1, 1, M, nz * nx)).astype(np.complex64))
    apod = torch.from_numpy(np.ascontiguousarray(ap.transpose(2, 1, 0).reshape(M, nz * nx)).astype(np.float32))
    out = postprocess.capon_minimum_variance(cube.to(cuda_dev), apod.to(cuda_dev), nz, nx, L, K, 1e-2,
                                             doForwardBackward=fb)
    want = O.capon_f64(d, ap, L, K, 1e-2, fb=fb)
    assert rel(out[0].cpu().numpy().reshape(nx, nz).T, want) <= 1e-3
