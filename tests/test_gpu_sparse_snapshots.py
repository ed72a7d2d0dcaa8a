"""Snapshots are stored only where they are non-zero: what an earlier circuit left in the buffer is never read."""

from __future__ import annotations

import pytest

import greenpeas_gb300 as gp
from conftest import compare_errors
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _text(n, rounds, dense):
    """n data qubits and measurements in one layout; dense: every error spreads over all of them."""
    t = "R " + " ".join(map(str, range(n))) + "\n"
    for r in range(rounds):
        t += "DEPOLARIZE2(0.001) " + " ".join(map(str, range(n))) + "\n"
        t += "".join(f"CX {q} {q + 1}\n" for q in range(n - 1)) if dense else "".join("TICK\n" for _ in range(n - 1))
        t += "X_ERROR(0.002) " + " ".join(map(str, range(n))) + "\nTICK\n"
        t += "M(0.003) " + " ".join(map(str, range(n))) + "\n"
        t += "".join(f"DETECTOR rec[-{k}]\n" for k in range(1, n + 1))
    return t


@pytest.mark.parametrize("kw", [{}, {"global_sort": True}, {"walk_segment": 4}, {"walk_words": 2}],
                         ids=["bucket", "global", "segments", "two_words"])
@pytest.mark.parametrize("n,rounds", [(2, 1), (8, 9), (34, 4), (66, 3)])
def test_dense_then_sparse(n, rounds, kw):
    dense, sparse = _text(n, rounds, True), _text(n, rounds, False)
    drv = gp.get_driver(dense, **kw)
    for text in (dense, sparse, dense, sparse):
        dem = drv.compile(text)
        compare_errors(dict(dem.errors()), dict(O.compile_text(text, 2).errors()), rel=1e-12)
