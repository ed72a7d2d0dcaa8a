"""Gradients of templates whose symptoms outgrow a bucket slot's targets and the target lists' first stride."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import compare_errors
from greenpeas_gb300 import noise as N
from greenpeas_gb300.autograd import NoiseRateDEM
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _template(span):
    """A flip of one qubit flips ``span`` neighbouring detectors, flips of a pair up to twice as many."""
    n = span + 40
    qs = " ".join(map(str, range(n)))
    text = f"R {qs}\nX_ERROR(0.001) {qs}\nTICK\nDEPOLARIZE1(0.001) {qs}\nTICK\nDEPOLARIZE2(0.001) "
    text += " ".join(f"{q} {q + n // 2}" for q in range(0, n // 2, 3)) + f"\nTICK\nM {qs}\n"
    return text + "".join("DETECTOR " + " ".join(f"rec[-{1 + (q + k) % n}]" for k in range(span)) + "\n" for q in range(n))


@pytest.mark.parametrize("span", [15, 16, 17, 26, 31, 32, 33, 64, 120, 130, 200])
def test_the_first_pass_is_right(span):
    """Forward and backward of a fresh template against the oracle: lists inside the slots, past them, and
    longer than the lists' stride (32, then 128), which the first forward widens; the next pass repeats it."""
    text = _template(span)
    model = NoiseRateDEM(text)
    rates = N.sample_rates(model.num_ticks, 5e-4, 2e-3, span)
    ref = O.compile_text(N.instantiate(text, rates), 2, provenance=True)
    w_ref = N.symptom_weights(ref.offsets, ref.targets, seed=1)
    g_ref = O.noise_gradient(ref, w_ref / np.array(ref.probs))
    assert max(len(t) for t, _ in ref.errors()) >= span
    first = None
    for _ in range(2):
        noise = torch.tensor(rates, dtype=torch.float64, device="cuda", requires_grad=True)
        p = model(noise)
        dem = model.last_dem()
        assert np.array_equal(p.detach().cpu().numpy(), dem.probs)
        compare_errors(dict(dem.errors()), dict(ref.errors()), rel=1e-12)
        w = N.symptom_weights(dem.offsets, dem.targets, seed=1)
        (torch.tensor(w, device="cuda") * torch.log(p)).sum().backward()
        g = noise.grad.cpu().numpy()
        assert np.all(np.abs(g - g_ref) <= 1e-10 * np.abs(g_ref) + 1e-13 * np.abs(g_ref).max())
        assert first is None or np.array_equal(g, first)
        first = g


def test_another_template_on_the_way():
    """Rates of one template are not taken for the next one's: short lists, long ones, short again."""
    for span in (5, 40, 5, 140):
        test_the_first_pass_is_right(span)
