"""Demodulation around the numbers of traces where CTAs begin to take several (a multiple of
the SMs' number) and where they are full, against the FP64 oracles at the bar of the kernel's
other tests; the first traces do not depend on how many follow."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import preprocess
from ustb_gb300.enums import Precision

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zero_phase", [False, True])
@pytest.mark.parametrize("L, D, ntaps", [(120, 2, 31), (645, 2, 31), (300, 1, 60), (2500, 1, 9)])
def test_numbers_of_traces(cuda_dev, L, D, ntaps, zero_phase):
    sms = torch.cuda.get_device_properties(cuda_dev).multi_processor_count
    rng = np.random.default_rng(L)
    fs, t0, fc = 20e6, 0.3e-6, 4.1e6
    rf = rng.standard_normal((20 * sms, L)).astype(np.float32)
    taps = np.hamming(ntaps + 2)[1:-1]
    taps = (taps / taps.sum()).astype(np.float32)
    x = torch.from_numpy(rf).to(cuda_dev)
    f = O.zero_phase_demodulation_f64 if zero_phase else O.fast_demodulation_f64
    want = f(rf[: 2 * sms + 1].T.astype(np.float64), fs, t0, fc, taps, D).T
    first = None
    for n in (1, sms - 1, sms, sms + 1, 2 * sms + 1, 7 * sms, 20 * sms):
        y = preprocess.demodulate(x[:n], fs, t0, fc, taps, D, Precision.fp32, 1.0, zero_phase=zero_phase)
        got = y.cpu().numpy()
        got = got[..., 0] + 1j * got[..., 1]
        m = min(n, 2 * sms + 1)
        assert np.linalg.norm(got[:m] - want[:m]) <= 1e-5 * np.linalg.norm(want[:m])
        first = y[0] if first is None else first
        assert torch.equal(y[0], first)
