"""The allocation-free merge at the bucket sizes where its paths change: a warp's 32, 64, 128 and 256 items, a block's
1,024, and the bucket past that."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from greenpeas_gb300 import _native

pytestmark = pytest.mark.gpu


def _merge(lists, p, stride):
    import torch

    n = len(lists)
    room = max(n, 1)  # (no null pointers)
    rows = np.zeros((room, stride), dtype=np.int32)
    for m, ts in enumerate(lists):
        rows[m, : len(ts)] = ts
    dev = torch.device("cuda", 0)
    tn = torch.tensor([len(ts) for ts in lists] + [0] * (room - n), dtype=torch.int32, device=dev)
    tl = torch.from_numpy(rows.reshape(-1)).to(dev)
    pr = torch.tensor(list(p) + [0.0] * (room - n), dtype=torch.float64, device=dev)
    cap = max(1, sum(map(len, lists)))
    out_p = torch.full((room,), -1.0, dtype=torch.float64, device=dev)
    off = torch.full((n + 1,), -1, dtype=torch.int32, device=dev)
    tg = torch.full((cap,), -1, dtype=torch.int32, device=dev)
    result = torch.zeros(4, dtype=torch.int32, device=dev)
    args = [ctypes.c_void_p(t.data_ptr()) for t in (tn, tl, pr, out_p, off, tg, result)]
    st = _native.lib().gpc_merge_mechanisms_static(args[0], args[1], stride, args[2], n, args[3], args[4], args[5], cap,
                                                   args[6], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    groups, targets, flags, _ = (int(x) for x in result.cpu())
    off, tg = off.cpu().numpy(), tg.cpu().numpy()
    assert int(off[groups]) == targets
    return flags, {tuple(int(t) for t in tg[off[g]:off[g + 1]]): float(out_p[g]) for g in range(groups)}, groups


def _expected(lists, p):
    runs = {}
    for ts, q in zip(lists, p):
        if ts:
            runs.setdefault(tuple(ts), []).append(q)
    return {ts: -float(np.expm1(np.log1p(-2 * np.array(qs)).sum())) / 2 for ts, qs in runs.items()}


@pytest.mark.parametrize("copies", [1, 31, 32, 33, 64, 65, 128, 129, 255, 256, 257, 600, 1020])
def test_one_symptom_many_times(copies):
    rng = np.random.default_rng(copies)
    lists = [[5, 70, 700]] * copies + [[int(a)] for a in rng.choice(5000, 40, replace=False)] + [[]]
    order = rng.permutation(len(lists))
    lists = [lists[k] for k in order]
    p = np.exp(rng.uniform(np.log(1e-6), np.log(1e-3), len(lists)))
    flags, got, groups = _merge(lists, p, 8)
    want = _expected(lists, p)
    assert flags == 0 and groups == len(want) and got.keys() == want.keys()
    assert all(abs(got[k] - want[k]) <= 1e-12 * want[k] for k in want)


def test_many_symptoms_in_long_and_short_runs():
    """2,000 symptoms of 1 to 60 mechanisms (about 60 to a bucket) of up to 12 targets, in every stride remainder."""
    rng = np.random.default_rng(3)
    sets = [sorted(int(t) for t in rng.choice(9000, int(rng.integers(1, 13)), replace=False)) for _ in range(2000)]
    lists = [s for s in sets for _ in range(int(rng.integers(1, 61)))]
    lists = [lists[k] for k in rng.permutation(len(lists))]
    p = np.exp(rng.uniform(np.log(1e-6), np.log(1e-3), len(lists)))
    flags, got, _ = _merge(lists, p, 12)
    want = _expected(lists, p)
    assert flags == 0 and got.keys() == want.keys()
    assert all(abs(got[k] - want[k]) <= 1e-12 * want[k] for k in want)


@pytest.mark.parametrize("n", [0, 1, 255, 257])
def test_small_inputs(n):
    lists = [[k % 7, 64 + k % 3] for k in range(n)]
    p = [1e-3] * n
    flags, got, groups = _merge(lists, p, 4)
    want = _expected(lists, p)
    assert flags == 0 and groups == len(want) and got.keys() == want.keys()
    assert all(abs(got[k] - want[k]) <= 1e-12 * want[k] for k in want)


def test_a_bucket_past_its_limit_is_reported():
    lists = [[3, 4]] * 1030 + [[9]] * 5
    flags, got, _ = _merge(lists, [1e-4] * len(lists), 4)
    assert flags == 16
    assert list(got) == [(9,)]
