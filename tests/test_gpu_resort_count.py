"""Re-sorts of the global path on more key bits are counted."""

from __future__ import annotations

import itertools

import numpy as np
import pytest

import greenpeas_gb300 as gp

pytestmark = pytest.mark.gpu


def _agreeing_pair(bits):
    """Two three-detector symptoms of word 0 whose keys agree on the top `bits` bits of the first half."""
    triples = list(itertools.combinations(range(64), 3))
    v = np.array([sum(1 << t for t in c) for c in triples], dtype=np.uint64)
    with np.errstate(over="ignore"):
        k = v * np.uint64(0x9E3779B97F4A7C15) + np.uint64(0xC2B2AE3D27D4EB4F)
        for c in (0xFF51AFD7ED558CCD, 0xC4CEB9FE1A85EC53):
            k = (k ^ (k >> np.uint64(33))) * np.uint64(c)
        top = (k ^ (k >> np.uint64(33))) >> np.uint64(64 - bits)
    order = np.argsort(top, kind="stable")
    i = int(np.flatnonzero(top[order][1:] == top[order][:-1])[0])
    return triples[order[i]], triples[order[i + 1]]


@pytest.mark.parametrize("agree", [False, True])
def test_a_sort_on_more_key_bits_is_counted(agree):
    """About 100 mechanisms sort on the top 24 key bits. Where two symptoms agree on them the first run sorts again
    on 64 bits, and the later ones start there: one re-sort over three runs, none where no two agree."""
    a, b = _agreeing_pair(24) if agree else ((0, 1, 2), (3, 4, 5))
    text = "R " + " ".join(map(str, range(66))) + "\n" + "X_ERROR(0.001) 64 65\nTICK\n" * 10
    text += "".join(f"CX 64 {t}\n" for t in a) + "".join(f"CX 65 {t}\n" for t in b)
    text += "X_ERROR(0.002) " + " ".join(map(str, range(64))) + "\nM " + " ".join(map(str, range(64))) + "\n"
    text += "".join(f"DETECTOR rec[-{64 - q}]\n" for q in range(64))
    drv = gp.get_driver(text, global_sort=True)
    drv.prepare(text)
    for _ in range(3):
        drv.run_device()
        drv.fetch()
    assert drv.fallback_counts()["full_key_resort"] == (1 if agree else 0)
