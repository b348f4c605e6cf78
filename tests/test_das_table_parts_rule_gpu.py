"""Table kernel on both sides of the numbers of pixels (in CTAs of 128 per SM), waves and
frames between which complex dimension.both stays in one part, against das_c's formula in
single precision (the das_c port; the parts add their sums in another order: 1e-5)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W, F", [(3, 1), (8, 1), (8, 2), (9, 1)])
@pytest.mark.parametrize("halves, extra", [(4, 1), (7, 0), (7, 1), (8, 0), (8, 1)])
def test_sides_of_the_rule(cuda_dev, W, F, halves, extra):
    sms = torch.cuda.get_device_properties(cuda_dev).multi_processor_count
    P, N, L = halves * sms * 64 + extra, 33, 128
    rng = np.random.default_rng(halves + W)
    fs, t0, fd = 20e6, 0.0, 5e6
    ch = (rng.standard_normal((L, N, W, F)) + 1j * rng.standard_normal((L, N, W, F))).astype(np.complex64)
    dtx, drx = (rng.uniform(0, 3e-6, (P, k)).astype(np.float32) for k in (W, N))
    atx = rng.uniform(0.2, 1, (P, W)).astype(np.float32)
    arx = rng.uniform(0, 1, (P, N)).astype(np.float32)
    arx[rng.random((P, N)) < 0.3] = 0
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).to(cuda_dev)  # noqa: E731
    out = kernels.das_table_f32(T(ch), fs, t0, T(atx), T(arx), T(dtx), T(drx), fd, 3).cpu().numpy().transpose(3, 2, 1, 0)
    want = O.das_f32(ch, np.float32(fs), np.float32(t0), atx, arx, dtx, drx, fd, 3)
    assert np.linalg.norm(out - want) <= 1e-5 * np.linalg.norm(want)
