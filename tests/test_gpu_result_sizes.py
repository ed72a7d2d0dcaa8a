"""A run's flags and sizes: from the emission where its blocks find their buckets' places, by a copy elsewhere."""

from __future__ import annotations

import pytest

import greenpeas_gb300 as gp
from greenpeas_gb300.codes import SurfaceCode

pytestmark = pytest.mark.gpu

EMPTY = "R 0\nM 0\nDETECTOR rec[-1]\n"
ONE = "R 0\nX_ERROR(0.01) 0\nM 0\nDETECTOR rec[-1]\n"
LONG = "R " + " ".join(map(str, range(700))) + "\n" + "".join(
    f"X_ERROR(0.001) {q}\n" for q in range(700)) + "M " + " ".join(map(str, range(700))) + "\n" + "".join(
    "DETECTOR " + " ".join(f"rec[-{1 + (q + k) % 700}]" for k in range(31)) + "\n" for q in range(700))


@pytest.fixture(scope="module")
def texts():
    return {"empty": EMPTY, "one": ONE, "long": LONG, "s3": SurfaceCode(3).get_memory(3, 1e-3, noise="uniform"),
            "s21": SurfaceCode(21).get_memory(21, 1e-3, noise="uniform")}


# bucket_mean 8 cuts the d = 21 circuit into 65,536 buckets, past the emission that writes the sizes itself
@pytest.mark.parametrize("kw", [{}, {"bucket_mean": 8}, {"bucket_mean": 128}, {"global_sort": True}],
                         ids=["table", "mean8", "mean128", "global"])
def test_sizes_follow_the_run(texts, kw):
    """One driver over circuits of all kinds, small after large and back: each run's sizes are its own, fetched
    or as device arrays, on the first runs and on replays."""
    want = {k: list(gp.get_driver(t).compile(t).errors()) for k, t in texts.items()}
    drv = gp.get_driver(texts["one"], **kw)
    for name in ("s21", "empty", "s3", "long", "one", "s21", "one", "s3"):
        drv.prepare(texts[name])
        for _ in range(3):
            drv.run_device()
            probs, offsets, _ = drv.device_dem()
            assert len(probs) == len(want[name])
            assert len(offsets) == len(want[name]) + 1
        got = dict(drv.fetch().errors())
        assert set(got) == {t for t, _ in want[name]}
        for t, p in want[name]:
            assert got[t] == pytest.approx(p, rel=1e-12)
