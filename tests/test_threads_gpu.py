"""Host threads that call one kernel with different amounts of shared memory at the same
time: every call succeeds and gives what it gives alone.  The C entries are called directly,
so that the threads spend most of their time in the library."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from ustb_gb300 import _lib, fast
from ustb_gb300.enums import Precision, Window
from ustb_gb300.geometry import Apodization
from ustb_gb300.uff import LinearScan, Probe, Wave

pytestmark = pytest.mark.gpu


def capon(dev, big):
    M = 64 if big else 8
    cube, apod = torch.randn(1, 1, M, 12, dtype=torch.complex64, device=dev), torch.ones(M, 12, device=dev)
    out = torch.empty(12, dtype=torch.complex64, device=dev)
    args = (cube.data_ptr(), apod.data_ptr(), 4, 3, M, 1, 4.0, 1, 1e-2, 0.16, 0, out.data_ptr())
    return "ustb_capon", args, out, (cube, apod)


def gcf(dev, big):
    K = 1024 if big else 300
    cube = torch.randn(1, 1, K, 64, dtype=torch.complex64, device=dev)
    out = torch.empty(64, device=dev)
    return "ustb_generalized_coherence", (cube.data_ptr(), 64, K, 1, 7, out.data_ptr(), None), out, cube


def demod(dev, big):
    n = 1001 if big else 9
    rf = torch.randn(4, 3000, device=dev)
    taps = torch.hann_window(n + 2, periodic=False, device=dev)[1:-1].contiguous()
    out = torch.empty(4, 1500, 2, device=dev)
    return "ustb_demodulate", (rf.data_ptr(), 0, out.data_ptr(), 0, 3000, 4, 20e6, 0.0, 5e6, 2, taps.data_ptr(), n,
                               1.0), out, (rf, taps)


def das(dev, big, batch=False):
    N, L = 400 if big else 8, 256
    probe = Probe.linear_array(N, 0.1e-3)
    scan = LinearScan(np.linspace(-1e-3, 1e-3, 8), np.linspace(5e-3, 6e-3, 8))
    g = fast.FastGeometry(probe, scan, [Wave.plane(0.0)], 20e6, 1e-6, 5e6, 1540.0, dev,
                          Apodization(window=Window.hanning, f_number=0.5), None)
    r = fast.Request(torch.randn(1, 1, N, L, 2, device=dev), Precision.fp32, True, g, 3, L=L)
    if batch:
        arr, scratch = (fast.CRequest * 1)(r.c_struct()), torch.zeros(2, dtype=torch.int64, device=dev)
        return "ustb_das_fast_batch", (ctypes.addressof(arr), 1, scratch.data_ptr()), r.outputs["cube"], (arr, scratch, r)
    flags = torch.zeros(1, dtype=torch.int32, device=dev)
    args = (r.ch.data_ptr(), 0, 1, L, N, 1, 1, ctypes.addressof(g.c), 3, 0, ctypes.addressof(r.c_out), flags.data_ptr())
    return "ustb_das_fast", args, r.outputs["cube"], (r, flags)


def das_batch(dev, big):
    return das(dev, big, True)


@pytest.mark.parametrize("make", [capon, gcf, demod, das, das_batch])
def test_threads(cuda_dev, make):
    torch.manual_seed(1)
    calls = [make(cuda_dev, i % 2) for i in range(4)]
    want = []
    for name, args, out, _ in calls:
        _lib.call(name, *args, torch.cuda.current_stream(cuda_dev).cuda_stream)
        torch.cuda.synchronize()
        want.append(out.clone())
    torch.cuda.synchronize()
    start, failed = threading.Barrier(len(calls)), []

    def work(i):
        name, args, out, _ = calls[i]
        entry, stream = getattr(_lib.lib(), name), torch.cuda.Stream(cuda_dev)
        torch.cuda.set_device(cuda_dev)
        start.wait()
        codes = [entry(*args, stream.cuda_stream) for _ in range(3000)]
        stream.synchronize()
        if any(codes) or not torch.equal(out, want[i]):
            failed.append((i, max(codes), sum(c != 0 for c in codes)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
