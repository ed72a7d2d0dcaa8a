"""The key pass merges a noise record's components of one symptom and keeps short target lists in the bucket slots:
records that need more words, values or targets than a warp holds, wide targets, long lists, and the bucket overflow."""

from __future__ import annotations

import pytest

import greenpeas_gb300 as gp
from conftest import compare_errors
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(dem, text, level=2):
    compare_errors(dict(dem.errors()), dict(O.compile_text(text, level).errors()), rel=1e-12)


def _fan(n, targets, noise):
    """Noise on the last qubits of n, each then copied onto its own list of qubits, which are measured."""
    src = range(n, n + len(targets))
    text = "R " + " ".join(map(str, range(n + len(targets)))) + "\n" + noise.format(*src) + "\n"
    for q, ts in zip(src, targets):
        text += "".join(f"CX {q} {t}\n" for t in ts)
    text += "DEPOLARIZE1(0.003) " + " ".join(map(str, range(0, n, 7))) + "\nM " + " ".join(map(str, range(n))) + "\n"
    return text + "".join(f"DETECTOR rec[-{n - q}]\n" for q in range(n))


def _deep(rounds, ancillas, detectors_each=1):
    """One data qubit copied onto fresh ancillas every round: an early error flips a detector of every later round."""
    n = ancillas
    anc = " ".join(map(str, range(1, n + 1)))
    body = f"R {anc}\nX_ERROR(0.0004) 1\n" + "".join(f"CX 0 {a}\n" for a in range(1, 1 + detectors_each)) + f"M {anc}\n"
    body += "".join(f"DETECTOR rec[-{k}]\n" for k in range(n, 0, -1)) + "TICK\n"
    return ("R 0\nDEPOLARIZE1(0.01) 0\nX_ERROR(0.002) 0\n" + f"REPEAT {rounds} {{\n{body}}}\n"
            + "DEPOLARIZE2(0.004) 0 1\nM 0 1\nDETECTOR rec[-1]\nOBSERVABLE_INCLUDE(0) rec[-2]\n")


def _cases():
    a, b = range(0, 200, 10), range(5, 200, 10)  # 20 targets each, in four words
    return {
        "union_of_40_targets": _fan(200, [a, b], "DEPOLARIZE2(0.01) {0} {1}\nDEPOLARIZE2(0.02) {1} {0}"),
        "union_of_32_targets": _fan(200, [list(a)[:16], list(b)[:16]], "DEPOLARIZE2(0.01) {0} {1}"),
        "lists_of_16_and_17": _fan(64, [range(16), range(20, 37)], "X_ERROR(0.01) {0} {1}\nX_ERROR(0.02) {0} {1}"),
        "shared_targets": _fan(96, [range(0, 90, 9), range(0, 90, 6)], "DEPOLARIZE2(0.01) {0} {1}\nPAULI_CHANNEL_1(0.01,0.02,0.03) {0}"),
        "words_65": _deep(70, 64),
        "words_64_exactly": _deep(63, 64),
        "wide_targets": _deep(1040, 64, 0),
    }


@pytest.mark.parametrize("name", ["union_of_40_targets", "union_of_32_targets", "lists_of_16_and_17", "shared_targets",
                                  "words_65", "words_64_exactly", "wide_targets"])
@pytest.mark.parametrize("level", [0, 1, 2])
def test_against_the_oracle(name, level):
    text = _cases()[name]
    _check(gp.get_driver(text, correlation_level=level).compile(text), text, level)


def test_a_batch_with_wide_targets_gives_the_single_dems():
    """One circuit of more than 65,536 detectors makes the whole batch's slots wide."""
    texts = [gp.SurfaceCode(5).get_memory(5, 1e-3, noise="uniform"), _cases()["wide_targets"],
             gp.BBCode(6).get_memory(3, 1e-3, noise="uniform"), _cases()["lists_of_16_and_17"]]
    singles = [gp.get_driver(t).compile(t) for t in texts]
    assert gp.get_driver(texts[0]).compile_batch(texts) == singles


@pytest.mark.parametrize("copies, overflows", [(127, False), (128, False), (129, True), (200, True)])
def test_a_bucket_overflows_by_its_mechanisms(copies, overflows):
    """X and Y of a channel whose Z is not detected are one item of two mechanisms: 128 copies fill a bucket."""
    text = "R 0 1\n" + "DEPOLARIZE1(0.0001) 0\nTICK\n" * copies + "CX 0 1\nM 0 1\nDETECTOR rec[-1]\nDETECTOR rec[-2]\n"
    drv = gp.get_driver(text)
    _check(drv.compile(text), text)
    assert drv.fallback_counts()["global_sort"] == (1 if overflows else 0)
