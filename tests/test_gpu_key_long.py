"""Records of long symptoms in the key pass: worked on side by side, with the same results in any company."""

from __future__ import annotations

import pytest

import greenpeas_gb300 as gp
from conftest import compare_errors
from oracle import oracle as O

pytestmark = pytest.mark.gpu

NOISE = {"x": "X_ERROR(0.001) {qs}\n", "1": "DEPOLARIZE1(0.002) {qs}\n", "2": "DEPOLARIZE2(0.003) {pairs}\n",
         "mixed": "X_ERROR(0.001) {qs}\nDEPOLARIZE1(0.002) {qs}\nDEPOLARIZE2(0.003) {pairs}\nX_ERROR(0.002) 0\n"
                  "DEPOLARIZE2(0.001) 0 1\nDEPOLARIZE1(0.001) 1\nPAULI_CHANNEL_1(0.01,0.02,0.03) 0\n"}


def _unreset(n, rounds, noise, apart=1):
    """n qubits measured every round without a reset, each measurement a detector: a flip shows in every later
    round.  Pairs are ``apart`` qubits apart (the same words of detectors, or others)."""
    qs = " ".join(map(str, range(n)))
    pairs = " ".join(f"{q} {(q + apart) % n}" for q in range(n))
    body = NOISE[noise].format(qs=qs, pairs=pairs) + f"TICK\nM {qs}\n"
    return f"R {qs}\n" + (body + "".join(f"DETECTOR rec[-{n - q}]\n" for q in range(n))) * rounds


def _check(text, level):
    dem = gp.get_driver(text, correlation_level=level).compile(text)
    compare_errors(dict(dem.errors()), dict(O.compile_text(text, level).errors()), rel=1e-12)
    return dem


# words a record: 8 to 66 (64 at once fit the other way), targets: 8 to 132 (32 a record fit it)
@pytest.mark.parametrize("noise", list(NOISE))
@pytest.mark.parametrize("level", [0, 1, 2])
@pytest.mark.parametrize("n, rounds, apart", [(70, 8, 1), (64, 33, 1), (70, 33, 35), (65, 64, 1), (64, 66, 31), (3, 40, 1)])
def test_against_the_oracle(n, rounds, apart, level, noise):
    _check(_unreset(n, rounds, noise, apart), level)


@pytest.mark.parametrize("level", [0, 2])
def test_in_a_batch_as_alone(level):
    """A batch's warps take other runs of records than a single circuit's: the DEMs are the same, bit for bit."""
    texts = [_unreset(40, 20, "mixed"), gp.SurfaceCode(5).get_memory(5, 1e-3, noise="uniform"), _unreset(9, 32, "mixed", 4),
             _unreset(64, 12, "1"), gp.BBCode(6).get_memory(6, 1e-3, noise="uniform"), _unreset(33, 15, "2", 16)]
    singles = [gp.get_driver(t, correlation_level=level).compile(t) for t in texts]
    assert gp.get_driver(texts[0], correlation_level=level).compile_batch(texts) == singles


def test_takes_no_longer_than_its_words():
    """The key pass beside the walk, which follows the same symptoms (one record at a time: 54 times its time)."""
    text = _unreset(400, 100, "mixed")
    drv = gp.get_driver(text)
    drv.set_stage_timing(True)
    drv.prepare(text)
    times = []
    for _ in range(6):
        drv.run_device()
        drv.device_dem()
        times.append(drv.last_timings())
    assert min(t["key"] for t in times) < 15 * min(t["walk"] for t in times)
