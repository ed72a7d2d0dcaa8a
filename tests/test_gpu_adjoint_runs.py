"""Gradients through runs of repeated symptoms: runs inside 32 sorted positions, across them and of merged components."""

from __future__ import annotations

import numpy as np
import pytest

import greenpeas_gb300 as gp
from greenpeas_gb300 import noise as N
from greenpeas_gb300.autograd import NoiseRateDEM
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("level", [0, 2])
@pytest.mark.parametrize("copies", [1, 2, 31, 32, 33, 63, 64, 65, 100, 125])
def test_repeated_symptoms(copies, level):
    """`copies` ticks of flips and of a channel whose Z is not detected (its X and Y merge), beside other symptoms."""
    text = "R 0 1 2 3\n" + "X_ERROR(0.001) 0\nDEPOLARIZE1(0.001) 0 1\nTICK\n" * (copies // 3 + 1)
    text += "X_ERROR(0.002) 1\nTICK\n" * copies + "DEPOLARIZE2(0.003) 0 2 1 3\nTICK\nCX 0 2\nDEPOLARIZE2(0.001) 0 2\nTICK\n"
    text += "X_ERROR(0.002) 0 1 2 3\nM 0 1 2 3\n" + "".join(f"DETECTOR rec[-{k}]\n" for k in range(4, 0, -1))
    model = NoiseRateDEM(text, correlation_level=level)
    rates = N.sample_rates(model.num_ticks, 5e-4, 2e-3, copies)
    noise = torch.tensor(rates, dtype=torch.float64, device="cuda", requires_grad=True)
    p = model(noise)
    dem = model.last_dem()
    w = N.symptom_weights(dem.offsets, dem.targets, seed=1)
    loss = (torch.tensor(w, device="cuda") * torch.log(p)).sum()
    try:
        loss.backward()
    except gp.GpcError as e:
        assert e.status == -3  # the two long runs fell into one bucket: the global sort has no gradients
        pytest.skip("more than a bucket's mechanisms")
    g = noise.grad.cpu().numpy()
    ref = O.compile_text(N.instantiate(text, rates), level, provenance=True)
    w_ref = N.symptom_weights(ref.offsets, ref.targets, seed=1)
    g_ref = O.noise_gradient(ref, w_ref / np.array(ref.probs))
    assert np.all(np.abs(g - g_ref) <= 1e-10 * np.abs(g_ref) + 1e-13 * np.abs(g_ref).max())
