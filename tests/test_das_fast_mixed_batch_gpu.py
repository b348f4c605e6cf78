"""Batches whose requests differ in storage type and number of waves: one launch while they
are few, and every request's own result (the batch's persistent kernel against a launch of
its own; 1e-6 leaves room for another order of the sums)."""
import numpy as np
import pytest
import torch

from ustb_gb300 import fast
from ustb_gb300.enums import Precision, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan, Probe, Wave

pytestmark = pytest.mark.gpu

L, FS, F0, T0 = 400, 20e6, 5e6, 2e-6


def request(rng, precision, W, cplx, dim, epi, dev, F=1, shape=0):
    N = 18
    seq = [Wave.plane(float(a)) for a in np.deg2rad(np.linspace(-9, 9, W))]
    scan = LinearScan(np.linspace(-3e-3, 3e-3, 23), np.linspace(6e-3, 11e-3, 47))
    rx = Apodization(window=Window.tukey25, f_number=1.2)
    g = fast.FastGeometry(Probe.linear_array(N, 0.3e-3), scan, seq, FS, T0, F0 if cplx else 0.0, 1540.0, dev, rx, None,
                          stage_shape=shape)
    x = rng.standard_normal((F, W, N, L) + ((2,) if cplx else ())).astype(np.float32)
    st = torch.from_numpy(x).to(dev).to(fast.TORCH_STORE[precision])
    return fast.Request(st, precision, cplx, g, dim, F=F, L=L, epilogue=epi)


def launches(scratch):
    return int((scratch[1:] != 0).sum())  # each launch has its own queue counter


@pytest.mark.parametrize("workspace", [False, True])
@pytest.mark.parametrize("dim, cplx, epi", [(3, True, False), (3, False, False), (2, True, False), (2, True, True),
                                            (1, True, False), (1, False, False), (0, True, False)])
def test_few_items_share_a_launch(cuda_dev, dim, cplx, epi, workspace):
    rng = np.random.default_rng(dim)
    reqs = [request(rng, p, W, cplx, dim, epi, cuda_dev, F=1 + W % 2)
            for p in (Precision.fp16, Precision.fp32, Precision.bf16) for W in (1, 2, 5, 11)]
    ws = torch.empty(fast.workspace_bytes(reqs), dtype=torch.uint8, device=cuda_dev) if workspace else None
    scratch = fast.das_fast_batch(reqs, workspace=ws)
    assert launches(scratch) == 1 and int(scratch[0]) == 0
    for r in reqs:
        alone = fast.das_fast(r.ch, r.precision, cplx, r.geom, dim, F=r.F, L=L, epilogue=epi)
        for k, y in r.outputs.items():
            ok = torch.isfinite(alone[k].abs())  # a factor is infinite where no weight exceeds the threshold
            assert torch.equal(ok, torch.isfinite(y.abs()))
            assert torch.linalg.vector_norm((y - alone[k])[ok]) <= 1e-6 * torch.linalg.vector_norm(alone[k][ok]), k


@pytest.mark.parametrize("cplx, dim, asked, expect", [(False, 3, 1, 2), (True, 1, 1, 1), (True, 3, 3, 1), (True, 2, 3, 1)])
def test_stages_asked_for(cuda_dev, cplx, dim, asked, expect):
    """A request of real data with a stage shape of its own keeps it, in a launch of its own;
    complex data takes the library's."""
    rng = np.random.default_rng(9)
    reqs = [request(rng, Precision.fp32, W, cplx, dim, False, cuda_dev, shape=s)
            for W, s in ((1, 0), (20, 0), (5, asked))]
    assert launches(fast.das_fast_batch(reqs, max_ctas=4)) == expect  # (bounded: persistent)
    for r in reqs:
        alone = fast.das_fast(r.ch, r.precision, cplx, r.geom, dim, L=L)["cube"]
        assert torch.linalg.vector_norm(r.outputs["cube"] - alone) <= 1e-6 * torch.linalg.vector_norm(alone)


def test_library_stages_asked_for_share(cuda_dev):
    """The shape that the library would choose, asked for (as tuned plans do)."""
    rng = np.random.default_rng(10)
    reqs = [request(rng, p, 5, True, 3, False, cuda_dev, shape=s)
            for p, s in ((Precision.fp16, 0), (Precision.fp32, 2), (Precision.bf16, 2))]
    assert launches(fast.das_fast_batch(reqs)) == 1


def test_many_items_keep_their_variants(cuda_dev):
    rng = np.random.default_rng(9)
    reqs = [request(rng, p, 1 + i % 2 * 3, True, 1, False, cuda_dev, F=600) for i in range(2) for p in (Precision.fp32,)]
    assert launches(fast.das_fast_batch(reqs)) == 2


@pytest.mark.parametrize("dim, cplx, epi", [(3, True, False), (3, False, False), (2, True, False), (2, False, False),
                                            (2, True, True), (1, True, False), (1, False, False)])
@pytest.mark.parametrize("precision", [Precision.fp32, Precision.fp16])
@pytest.mark.parametrize("W, F", [(1, 1), (20, 2), (75, 3), (3, 400)])
def test_one_small_request(cuda_dev, W, F, precision, dim, cplx, epi):
    """Fewer work items than SMs: a grid launch in parts where that is faster, with scratch
    from the pool or from what a workspace has left; with a bound on the CTAs, and with many
    frames, the persistent one.  The same result every way, and every time."""
    rng = np.random.default_rng(W)
    r = request(rng, precision, W, cplx, dim, epi, cuda_dev, F=F)
    alone = fast.das_fast(r.ch, r.precision, cplx, r.geom, dim, F=F, L=L, epilogue=epi)
    bytes_ = fast.workspace_bytes([r])
    for extra, max_ctas in ((None, 0), (0, 0), (1 << 22, 0), (0, 3)):
        ws = None if extra is None else torch.empty(bytes_ + extra, dtype=torch.uint8, device=cuda_dev)
        counts = []
        for _ in range(2):
            scratch = fast.das_fast_batch([r], workspace=ws, max_ctas=max_ctas)
            assert int(scratch[0]) == 0
            counts.append(launches(scratch))
        assert counts[0] == counts[1] and (counts[0] == 1 or (max_ctas == 0 and F < 400))
        if W == 75 and extra != 0:
            assert counts[0] == 0  # a grid launch has no queue counter
        for k, y in r.outputs.items():
            ok = torch.isfinite(alone[k].abs())
            assert torch.equal(ok, torch.isfinite(y.abs()))
            bar = 1e-6 if k == "cube" else 1e-5  # the factors square and divide sums of another order
            assert torch.linalg.vector_norm((y - alone[k])[ok]) <= bar * torch.linalg.vector_norm(alone[k][ok]), k
