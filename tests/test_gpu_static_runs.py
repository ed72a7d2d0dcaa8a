"""The allocation-free merge on few symptoms of many copies each: what its buckets of 257 to 1,024 items cost."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from greenpeas_gb300 import _native

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _best(symptoms, copies, stride=8):
    """Time (ms) of merging ``symptoms`` pairs of targets, ``copies`` mechanisms each, in mixed order."""
    n = symptoms * copies
    rows = np.zeros((n, stride), dtype=np.int32)
    which = np.random.default_rng(1).permutation(n) % symptoms
    rows[:, 0], rows[:, 1] = 3 * which, 3 * which + 100000
    dev = torch.device("cuda", 0)
    tn = torch.full((n,), 2, dtype=torch.int32, device=dev)
    tl, p = torch.from_numpy(rows.reshape(-1)).to(dev), torch.full((n,), 1e-4, dtype=torch.float64, device=dev)
    out_p, off = torch.zeros(n, dtype=torch.float64, device=dev), torch.zeros(n + 1, dtype=torch.int32, device=dev)
    tg, result = torch.zeros(2 * n, dtype=torch.int32, device=dev), torch.zeros(4, dtype=torch.int32, device=dev)
    args = [ctypes.c_void_p(t.data_ptr()) for t in (tn, tl, p, out_p, off, tg, result)]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    times = []
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        _native.check(_native.lib().gpc_merge_mechanisms_static(args[0], args[1], stride, args[2], n, args[3], args[4],
                                                                args[5], 2 * n, args[6], stream))
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    assert result.tolist()[:3] == [symptoms, 2 * symptoms, 0]
    want = 0.5 * (1 - (1 - 2e-4) ** copies)
    assert np.allclose(out_p[:symptoms].cpu().numpy(), want, rtol=1e-12)
    return min(times)


def test_long_runs_beside_short_ones():
    """Buckets of 900 equal items against the same number of mechanisms in pairs (with a pass over the bucket for
    each item of a thread: over 15 times the time)."""
    assert _best(10, 900) < 10 * _best(4500, 2)
