"""The global sort path: runs that cross merge tiles, and the top-bits sort that two keys can share."""

from __future__ import annotations

import itertools

import numpy as np
import pytest

import greenpeas_gb300 as gp
from conftest import compare_errors
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(dem, text):
    compare_errors(dict(dem.errors()), dict(O.compile_text(text, 2).errors()), rel=1e-12)


@pytest.mark.parametrize("copies", [(1, 1), (31, 33), (255, 257), (256, 256), (300, 212), (511, 1), (513, 767), (2000, 40)])
def test_runs_across_merge_tiles(copies):
    """Runs of equal symptoms that end before, at and after tile boundaries (256 sorted positions), run twice:
    the second run of a prepared circuit whose bucket overflowed goes to the sort at once."""
    a, b = copies
    text = "R 0 1 2 3\n" + "X_ERROR(0.0003) 0\nTICK\n" * a + "X_ERROR(0.0002) 1\nTICK\n" * b
    text += "DEPOLARIZE1(0.001) 2 3\nDEPOLARIZE2(0.001) 0 2 1 3\nM 0 1 2 3\n"
    text += "".join(f"DETECTOR rec[-{k}]\n" for k in range(1, 5))
    _check(gp.get_driver(text, global_sort=True).compile(text), text)
    drv = gp.get_driver(text)
    drv.prepare(text)
    dems = []
    for _ in range(2):
        drv.run_device()
        dems.append(drv.fetch())
    _check(dems[0], text)
    assert dems[0] == dems[1]
    small = "R 0\nX_ERROR(0.01) 0\nM 0\nDETECTOR rec[-1]\n"
    _check(drv.compile(small), small)  # the next circuit starts on the bucket path again


def _top_bits(v, bits):
    """Top bits of a one-word symptom's first key half (word 0)."""
    def mix(k):
        for c in (0xFF51AFD7ED558CCD, 0xC4CEB9FE1A85EC53):
            k = (k ^ (k >> np.uint64(33))) * np.uint64(c)
        return k ^ (k >> np.uint64(33))
    with np.errstate(over="ignore"):
        return mix(v * np.uint64(0x9E3779B97F4A7C15) + np.uint64(0xC2B2AE3D27D4EB4F)) >> np.uint64(64 - bits)


def test_two_symptoms_that_agree_on_the_sorted_bits():
    """A circuit of ~100 mechanisms sorts on the top 24 key bits; two of its symptoms agree on them and
    their copies alternate, so the merge must notice and sort on all 64 bits."""
    triples = list(itertools.combinations(range(64), 3))
    v = np.array([sum(1 << t for t in c) for c in triples], dtype=np.uint64)
    top = _top_bits(v, 24)
    order = np.argsort(top, kind="stable")
    k = int(np.flatnonzero(top[order][1:] == top[order][:-1])[0])
    a, b = triples[order[k]], triples[order[k + 1]]
    text = "R " + " ".join(map(str, range(66))) + "\n" + "X_ERROR(0.001) 64 65\nTICK\n" * 10
    text += "".join(f"CX 64 {t}\n" for t in a) + "".join(f"CX 65 {t}\n" for t in b)
    text += "X_ERROR(0.002) " + " ".join(map(str, range(64))) + "\nM " + " ".join(map(str, range(64))) + "\n"
    text += "".join(f"DETECTOR rec[-{64 - q}]\n" for q in range(64))
    dem = gp.get_driver(text, global_sort=True).compile(text)
    assert {a, b} <= {t for t, _ in dem.errors()}
    _check(dem, text)


def test_later_runs_of_such_a_circuit_sort_on_64_bits():
    """The next run of that circuit starts on 64 bits: same result; the driver's next circuit is not bound by it."""
    triples = list(itertools.combinations(range(64), 3))
    v = np.array([sum(1 << t for t in c) for c in triples], dtype=np.uint64)
    top = _top_bits(v, 24)
    order = np.argsort(top, kind="stable")
    k = int(np.flatnonzero(top[order][1:] == top[order][:-1])[0])
    a, b = triples[order[k]], triples[order[k + 1]]
    text = "R " + " ".join(map(str, range(66))) + "\n" + "X_ERROR(0.001) 64 65\nTICK\n" * 10
    text += "".join(f"CX 64 {t}\n" for t in a) + "".join(f"CX 65 {t}\n" for t in b)
    text += "X_ERROR(0.002) " + " ".join(map(str, range(64))) + "\nM " + " ".join(map(str, range(64))) + "\n"
    text += "".join(f"DETECTOR rec[-{64 - q}]\n" for q in range(64))
    drv = gp.get_driver(text, global_sort=True)
    drv.prepare(text)
    dems = []
    for _ in range(3):
        drv.run_device()
        dems.append(drv.fetch())
    _check(dems[0], text)
    assert dems[0] == dems[1] == dems[2]
    small = "R 0 1\nX_ERROR(0.01) 0\nX_ERROR(0.02) 1\nM 0 1\nDETECTOR rec[-1]\nDETECTOR rec[-2]\n"
    _check(drv.compile(small), small)


@pytest.mark.parametrize("forced", [False, True])
@pytest.mark.parametrize("copies", [300, 4000])
def test_repeated_runs_take_a_graph(forced, copies):
    """Runs of a prepared circuit on the global path (the third and later ones replay a graph), then another
    circuit of the same driver and the first one again."""
    def text(p):
        t = "R 0 1 2 3\n" + f"X_ERROR({p}) 0\nTICK\n" * copies + "DEPOLARIZE2(0.001) 0 2 1 3\nM 0 1 2 3\n"
        return t + "".join(f"DETECTOR rec[-{k}]\n" for k in range(1, 5))
    drv = gp.get_driver(text(0.0001), global_sort=forced)
    for p in (0.0001, 0.0002, 0.0001):  # the same sizes: one graph serves them all
        drv.prepare(text(p))
        dems = []
        for _ in range(5):
            drv.run_device()
            dems.append(drv.fetch())
        _check(dems[0], text(p))
        assert all(d == dems[0] for d in dems)
    small = "R 0\nX_ERROR(0.01) 0\nM 0\nDETECTOR rec[-1]\n"
    _check(drv.compile(small), small)
