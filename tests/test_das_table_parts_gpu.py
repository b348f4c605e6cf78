"""The table kernel with four warps to a pixel's channels (few pixels) against one thread
per pixel (many): the same 333 pixels alone and repeated beyond the line between the two.
Up to 680 units are summed in two orders, which differ by about sqrt(680) * 2^-24 = 1.6e-6;
the bar is 2e-6.  Channels without a weight at both ends, warps without any."""
import numpy as np
import pytest
import torch

from ustb_gb300 import kernels

pytestmark = pytest.mark.gpu

P = 333


@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("dim", [0, 1, 2, 3])
@pytest.mark.parametrize("W, N, F", [(1, 32, 1), (2, 37, 2), (6, 33, 5), (17, 40, 1)])
def test_parts(cuda_dev, W, N, F, dim, cplx):
    rng = np.random.default_rng(W * 100 + N + dim)
    L, reps = 190, 10 * 152 * 128 // P + 1
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(cuda_dev)
    x = T(rng.standard_normal((F, W, N, L) + ((2,) if cplx else ())))
    x = torch.view_as_complex(x) if cplx else x
    dtx, drx = T(rng.uniform(0, 5e-6, (W, P))), T(rng.uniform(0, 7e-6, (N, P)))
    atx, arx = rng.uniform(0.2, 1, (W, P)), rng.uniform(0.1, 1, (N, P))
    atx[rng.random((W, P)) < 0.1] = 0
    arx[rng.random((N, P)) < 0.3] = 0
    arx[: N // 5, :100] = 0
    arx[-N // 4:, 50:200] = 0
    arx[:, 64:130] = 0  # whole warps without a receive weight
    atx, arx = T(atx), T(arx)
    run = lambda r: kernels.das_table_f32(x, 20e6, 1e-6, *(t.repeat(1, r) for t in (atx, arx, dtx, drx)),
                                          5e6 if cplx else 0.0, dim)
    few, many = run(1), run(reps)[..., -P:]
    assert torch.isfinite(torch.view_as_real(few) if cplx else few).all()
    assert torch.linalg.vector_norm(few - many) <= 2e-6 * torch.linalg.vector_norm(many)
    assert torch.equal(few == 0, many == 0)
