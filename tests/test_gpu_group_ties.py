"""Buckets filled by few symptoms repeated many times: their order, and that it costs no more than its items."""

from __future__ import annotations

import pytest

import greenpeas_gb300 as gp
from conftest import compare_errors
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _copies(counts):
    """``counts[q]`` flips of qubit q, at rates of their own, every qubit read by a detector."""
    n = len(counts)
    text = "R " + " ".join(map(str, range(n))) + "\n"
    for k in range(max(counts)):
        qs = [q for q in range(n) if counts[q] > k]
        text += f"X_ERROR({1e-4 * (1 + k % 17)}) " + " ".join(map(str, qs)) + "\nTICK\n"
    return text + "M " + " ".join(map(str, range(n))) + "\n" + "".join(f"DETECTOR rec[-{n - q}]\n" for q in range(n))


@pytest.mark.parametrize("counts", [(32,), (33,), (63, 1), (64,), (65, 40), (127, 1), (128,), (129, 100), (255,), (256,),
                                    (200, 56, 1, 2), (31, 1, 33, 2, 64, 3, 17, 90, 5)])
@pytest.mark.parametrize("mean", [8, 128])
def test_runs_across_the_sorted_chunks(counts, mean):
    """Runs of equal symptoms that end before, at and after every 32 positions of a bucket's order."""
    text = _copies(counts)
    drv = gp.get_driver(text, bucket_mean=mean)
    dem = drv.compile(text)
    compare_errors(dict(dem.errors()), dict(O.compile_text(text, 2).errors()), rel=1e-12)
    assert dem == drv.compile(text)


def test_repeated_symptoms_take_no_longer_than_others():
    """The grouping beside the walk (64 us to 8; every item searching along its run: 307)."""
    text = _copies([250] * 40)
    drv = gp.get_driver(text)
    drv.set_stage_timing(True)
    drv.prepare(text)
    times = []
    for _ in range(6):
        drv.run_device()
        drv.device_dem()
        times.append(drv.last_timings())
    assert drv.fallback_counts()["global_sort"] == 0
    assert min(t["sort"] for t in times) < 16 * min(t["walk"] for t in times)
