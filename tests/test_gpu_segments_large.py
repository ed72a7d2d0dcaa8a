"""The segmented walk's instances: two qubits per thread, one, two and four transfer columns per CTA."""

from __future__ import annotations

import pytest

import greenpeas_gb300 as gp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d, rounds, qpt", [(7, 7, 2), (9, 3, 1), (15, 6, 1), (17, 6, 1), (17, 6, 2), (23, 6, 2)])
@pytest.mark.parametrize("target", [12, 40, 96])
def test_equals_the_plain_walk(d, rounds, qpt, target):
    """Surface memories of 128 to 1,100 slots (d = 17: 900, d = 23: two qubits per thread by size), cut at several
    densities, against the plain walk: the same DEM, bit for bit, fresh and from a captured graph."""
    text = gp.SurfaceCode(d).get_memory(rounds, 2e-3, noise="uniform")
    plain = gp.get_driver(text, walk_segment=-1).compile(text)
    drv = gp.get_driver(text, walk_segment=target, walk_qpt=qpt)
    drv.prepare(text)
    if drv.walk_segments()["segments"] == 0:
        pytest.skip("too short to cut at this target, or the slots do not split over the threads")
    for _ in range(3):
        drv.run_device()
        assert drv.fetch() == plain
