"""Capon on both sides of 64 channels, where the kernel changes, against the FP64 oracle:
apertures whose numbers of subarrays lie around the blocks of 8 products that the first
window is summed in, one-sample and clipped depth windows.  The bar is that of the kernel's
other tests."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import postprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, L", [(64, 32), (65, 32), (65, 1), (66, 2), (97, 31), (200, 8), (256, 32)])
@pytest.mark.parametrize("K, fb", [(0, False), (0, True), (4, False), (30, True)])
def test_both_sides_of_the_kernels(cuda_dev, M, L, K, fb):
    rng = np.random.default_rng(M + L + K)
    nz, nx = 12, 3
    d = 0.3 * (rng.standard_normal((nz, nx, M)) + 1j * rng.standard_normal((nz, nx, M)))
    d += np.exp(1j * 0.3 * np.arange(M)) * rng.standard_normal((nz, nx, 1))
    ap = np.ones((nz, nx, M))
    for iz in range(nz):
        ap[iz, 1, iz:iz + M - 12] = 0  # gaps: more subarrays than active channels give
        ap[iz, 2, :M - 2 - iz] = 0     # a few channels at the end
    cube = torch.from_numpy(np.ascontiguousarray(d.transpose(2, 1, 0).reshape(1, 1, M, nz * nx)).astype(np.complex64))
    apod = torch.from_numpy(np.ascontiguousarray(ap.transpose(2, 1, 0).reshape(M, nz * nx)).astype(np.float32))
    out = postprocess.capon_minimum_variance(cube.to(cuda_dev), apod.to(cuda_dev), nz, nx, L, K, 1e-2,
                                             doForwardBackward=fb)
    want = O.capon_f64(d, ap, L, K, 1e-2, fb=fb)
    assert np.linalg.norm(out[0].cpu().numpy().reshape(nx, nz).T - want) <= 1e-3 * np.linalg.norm(want)
