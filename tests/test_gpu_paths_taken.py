"""The path a run takes where it is known beforehand: buckets that cannot overflow and walks that are cut."""

from __future__ import annotations

import pytest

import greenpeas_gb300 as gp
from greenpeas_gb300 import noise as N
from greenpeas_gb300.autograd import NoiseRateDEM

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("level", [0, 2])
@pytest.mark.parametrize("copies", [1, 2, 31, 32, 33])
def test_gradients_of_small_circuits_keep_the_bucket_merge(copies, level):
    """Circuits of at most 256 mechanisms fit any bucket: their gradients are never refused."""
    text = "R 0 1 2 3\n" + "X_ERROR(0.001) 0\nDEPOLARIZE1(0.001) 0 1\nTICK\n" * (copies // 3 + 1)
    text += "X_ERROR(0.002) 1\nTICK\n" * copies + "DEPOLARIZE2(0.003) 0 2 1 3\nTICK\nCX 0 2\nDEPOLARIZE2(0.001) 0 2\nTICK\n"
    text += "X_ERROR(0.002) 0 1 2 3\nM 0 1 2 3\n" + "".join(f"DETECTOR rec[-{k}]\n" for k in range(4, 0, -1))
    drv = gp.get_driver(text, gp.CorrelationLevel(level))
    drv.prepare(text)
    assert drv.last_sizes()["raw"] <= 256
    model = NoiseRateDEM(text, correlation_level=level)
    rates = N.sample_rates(model.num_ticks, 5e-4, 2e-3, copies)
    noise = torch.tensor(rates, dtype=torch.float64, device="cuda", requires_grad=True)
    model(noise).sum().backward()
    assert bool((noise.grad != 0).any())


@pytest.mark.parametrize("d, rounds, qpt", [(7, 7, 2), (9, 3, 1), (15, 6, 1), (17, 6, 1), (17, 6, 2), (23, 6, 2)])
@pytest.mark.parametrize("target", [12, 40, 96])
def test_long_walks_are_cut(d, rounds, qpt, target):
    """Walks that span at least two segments of `target` cost units are cut (three rounds are about 120 units)."""
    text = gp.SurfaceCode(d).get_memory(rounds, 2e-3, noise="uniform")
    drv = gp.get_driver(text, walk_segment=target, walk_qpt=qpt)
    drv.prepare(text)
    assert (drv.walk_segments()["segments"] >= 2) == (rounds > 3 or target < 96)
