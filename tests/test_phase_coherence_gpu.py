"""Phase coherence factors of values that are not numbers and of tapered weights, against
the FP64 oracle at the bar of the kernel's other tests."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ustb_gb300 import postprocess

pytestmark = pytest.mark.gpu


def factors(c, w, dev):
    """FCA and FCC [P] of values and weights [K, P]."""
    w = None if w is None else torch.from_numpy(w.astype(np.float32)).to(dev)
    got = postprocess.phase_coherence_factor(torch.from_numpy(c.astype(np.complex64)[None, None]).to(dev), w)
    return got["FCA"][0].cpu().numpy(), got["FCC"][0].cpu().numpy()


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("bad", [complex(np.nan, 1), complex(1, np.nan), complex(-1, np.nan), complex(np.nan, np.nan),
                                 complex(np.inf, np.nan)])
def test_values_that_are_not_numbers(cuda_dev, bad, weighted):
    """A NaN in either component: FCA 0 and FCC NaN for that pixel alone."""
    rng = np.random.default_rng(3)
    K, P = 21, 70
    c = rng.standard_normal((K, P)) + 1j * rng.standard_normal((K, P)) + 2
    c[np.arange(K), 3 * np.arange(K)] = bad  # each channel in a pixel of its own
    w = rng.uniform(0.1, 1, (K, P)) if weighted else None
    fca, fcc = factors(c, w, cuda_dev)
    want_a, want_c, _ = O.phase_coherence_factor_f64(c.T, None if w is None else w.T)
    assert np.array_equal(np.isnan(fcc), np.isnan(want_c)) and np.isnan(want_c).sum() == K
    assert np.max(np.abs(fca - want_a)) <= 1e-4


@pytest.mark.parametrize("light, spread", [(1e-3, 1e-3), (1e-5, 1e-3), (1e-7, 1e-3), (1e-7, 1e-4)])
@pytest.mark.parametrize("edge", [1, 4, 16])
def test_light_edges_away_from_the_rest(cuda_dev, edge, light, spread):
    """Phases that agree but for the aperture's edges, whose weights are small (a taper)."""
    rng = np.random.default_rng(edge)
    K, P = 64, 130
    ang = 1.0 + spread * rng.standard_normal((K, P))
    w = np.ones((K, P), np.float32)
    for k in (slice(0, edge), slice(K - edge, K)):
        ang[k] = -1.8
        w[k] = light
    c = np.exp(1j * ang).astype(np.complex64)
    fca, fcc = factors(c, w, cuda_dev)
    want_a, want_c, _ = O.phase_coherence_factor_f64(c.T, w.T.astype(np.float64))
    assert np.max(np.abs(fca - want_a)) <= 1e-4
    assert np.max(np.abs(fcc - want_c)) <= 1e-4
