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
