"""Grouping a bucket: sizes around a warp's registers and shared memory, and two keys that share the sorted word."""

from __future__ import annotations

import itertools

import numpy as np
import pytest

import greenpeas_gb300 as gp
from conftest import compare_errors
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _mix(k):
    for c in (0xFF51AFD7ED558CCD, 0xC4CEB9FE1A85EC53):
        k = (k ^ (k >> np.uint64(33))) * np.uint64(c)
    return k ^ (k >> np.uint64(33))


def _keys(v):
    """128-bit keys of one-word symptoms (word 0)."""
    v = np.asarray(v, dtype=np.uint64)
    with np.errstate(over="ignore"):
        return (_mix(v * np.uint64(0x9E3779B97F4A7C15) + np.uint64(0xC2B2AE3D27D4EB4F)),
                _mix(v * np.uint64(0xD6E8FEB86659FD93) + np.uint64(0xA0761D6478BD642F) + np.uint64(0x8EBC6AF09C88C6E3)))


def _check(text, bits):
    """The DEM against the oracle, and its order against the keys': bucket, top of the second half, first half."""
    dem = gp.get_driver(text).compile(text)
    compare_errors(dict(dem.errors()), dict(O.compile_text(text, 2).errors()), rel=1e-12)
    x, y = _keys([sum(1 << t for t in ts) for ts, _ in dem.errors()])
    order = np.lexsort((y, x, y >> np.uint64(58), x >> np.uint64(64 - bits)))
    assert np.array_equal(order, np.arange(len(x)))
    return dem


def _circuit(sources, noise):
    """64 measured qubits; source k (qubit 64 + k) is copied onto the qubits of sources[k] after the noise lines."""
    n = 64 + len(sources)
    text = "R " + " ".join(map(str, range(n))) + "\n" + noise
    for k, ts in enumerate(sources):
        text += "".join(f"CX {64 + k} {t}\n" for t in ts)
    text += "M " + " ".join(map(str, range(64))) + "\n"
    return text + "".join(f"DETECTOR rec[-{64 - q}]\n" for q in range(64))


@pytest.mark.parametrize("copies", [1, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 192, 255, 256])
def test_buckets_of_every_size(copies):
    """One symptom `copies` times, others of one to three mechanisms in the buckets beside it."""
    noise = "X_ERROR(0.0003) 64\nTICK\n" * copies + "X_ERROR(0.001) 65 66\n" * 2 + "X_ERROR(0.002) 66\n"
    text = _circuit([[3, 9], [1, 2, 40], [5]], noise)
    mechanisms = copies + 5
    _check(text, 4 if mechanisms <= 256 else 5)


def test_many_symptoms_in_few_buckets():
    """240 symptoms of several mechanisms each in 16 to 64 buckets: runs of every length, crossing 32 positions."""
    sets = list(itertools.combinations(range(64), 2))[::8][:240]
    noise = "".join("X_ERROR(0.0007) " + " ".join(str(64 + k) for k in range(len(sets)) if k % 7 >= r) + "\nTICK\n" for r in range(7))
    m = sum(len([k for k in range(len(sets)) if k % 7 >= r]) for r in range(7))
    bits = 4
    while 16 << bits < m:
        bits += 1
    _check(_circuit([list(s) for s in sets], noise), bits)


def test_two_keys_that_share_the_sorted_word():
    """Two symptoms of one bucket agree on the 24 key bits that are sorted; their copies alternate, so the order
    must come from the full keys."""
    sets = list(itertools.combinations(range(64), 4))
    v = np.array([sum(1 << t for t in c) for c in sets], dtype=np.uint64)
    x, y = _keys(v)
    word = (x >> np.uint64(64 - 24)) << np.uint64(6) | (y >> np.uint64(58))  # 24 bits of x, 6 of y
    order = np.argsort(word, kind="stable")
    k = int(np.flatnonzero(word[order][1:] == word[order][:-1])[0])
    a, b = int(order[k]), int(order[k + 1])
    # a third symptom of the same bucket (4 bits) that differs from them right after the bucket's bits
    c = int(np.flatnonzero(((x ^ x[a]) >> np.uint64(59)) == 1)[0])
    noise = "X_ERROR(0.001) 64 65\nTICK\nX_ERROR(0.002) 65 64 66\nTICK\n" * 9
    dem = _check(_circuit([sets[a], sets[b], sets[c]], noise), 4)
    assert dem.num_errors == 3
