"""The table kernel around the wave counts where its chunks change from channels to waves,
against the das_c port (1e-5, the table path's bar): every sum mode, real and complex,
one and several frames, channel counts around the chunk of 8, zero weights, traces that
end inside the delays."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("dim", [0, 1, 2, 3])
@pytest.mark.parametrize("W, N, F", [(1, 1, 1), (1, 16, 1), (2, 9, 3), (3, 7, 2), (4, 8, 5), (5, 23, 1), (6, 17, 1), (9, 3, 2)])
def test_few_waves(cuda_dev, W, N, F, dim, cplx):
    rng = np.random.default_rng(W * 100 + N + dim)
    L, P = 190, 333
    ch = rng.standard_normal((L, N, W, F)) + (1j * rng.standard_normal((L, N, W, F)) if cplx else 0)
    ch = ch.astype(np.complex64 if cplx else np.float32)
    fs, t0, fd = np.float32(20e6), np.float32(1e-6), np.float32(5e6 if cplx else 0.0)
    dtx = rng.uniform(0, 5e-6, (P, W)).astype(np.float32)
    drx = rng.uniform(0, 7e-6, (P, N)).astype(np.float32)
    atx = rng.uniform(0.2, 1, (P, W)).astype(np.float32)
    arx = rng.uniform(0, 1, (P, N)).astype(np.float32)
    atx[rng.random((P, W)) < 0.1] = 0
    arx[rng.random((P, N)) < 0.4] = 0
    arx[64:160] = 0  # whole warps without a receive weight
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).to(cuda_dev)
    x = torch.from_numpy(np.ascontiguousarray(ch.transpose(3, 2, 1, 0))).to(cuda_dev)
    out = kernels.das_table_f32(x, float(fs), float(t0), T(atx), T(arx), T(dtx), T(drx), float(fd), dim)
    got = out.cpu().numpy().transpose(3, 2, 1, 0)
    want = O.das_f32(ch.astype(np.complex64), fs, t0, atx, arx, dtx, drx, fd, dim)
    want = want if cplx else want.real
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 1e-5
    assert np.all(got[want == 0] == 0)
