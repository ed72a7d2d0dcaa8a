"""The device arrays of a run: tensors of their own, whatever mode the first call was made in, wherever the buffers lie."""

from __future__ import annotations

import io

import numpy as np
import pytest

import greenpeas_gb300 as gp
from greenpeas_gb300.codes import SurfaceCode

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _memory(d, p=1e-3):
    return SurfaceCode(d).get_memory(d, p, noise="uniform")


def test_a_first_call_in_inference_mode_does_not_bind_later_ones():
    text = _memory(3)
    drv = gp.get_driver(text)
    drv.prepare(text)
    drv.run_device()
    with torch.inference_mode():
        assert all(t.is_inference() for t in drv.device_dem())
    probs, offsets, targets = drv.device_dem()
    assert not any(t.is_inference() for t in (probs, offsets, targets))
    scale = torch.ones_like(probs, requires_grad=True)
    (grad,) = torch.autograd.grad((scale * probs).sum(), scale)
    assert torch.equal(grad, probs)


def test_each_array_has_its_own_storage():
    """Saving one circuit's arrays writes these arrays and not the run's buffers."""
    texts = [_memory(3), _memory(5), _memory(3, 2e-3)]
    drv = gp.get_driver(texts[0])
    drv.prepare_batch(texts)
    drv.run_device()
    for i in range(len(texts)):
        for t in drv.device_dem(i):
            assert t.untyped_storage().nbytes() == t.numel() * t.element_size()
            assert t.storage_offset() == 0 and t._base is None
    buf = io.BytesIO()
    probs = drv.device_dem(1)[0]
    torch.save(probs, buf)
    assert buf.tell() < probs.numel() * 8 + 4096


@pytest.mark.parametrize("sizes", [(3, 9), (9, 3), (3, 9, 3, 13)])
def test_values_after_the_buffers_moved(sizes):
    """Circuits small after large and back on one driver: the arrays hold what fetch() returns."""
    drv = gp.get_driver(_memory(sizes[0]))
    for k, d in enumerate(sizes):
        drv.prepare(_memory(d, 1e-3 * (k + 1)))
        for _ in range(3):
            drv.run_device()
            probs, offsets, targets = (t.cpu().numpy() for t in drv.device_dem())
            dem = drv.fetch()
            assert np.array_equal(probs, dem.probs)
            assert np.array_equal(offsets, np.asarray(dem.offsets).astype(np.int32))
            assert np.array_equal(targets, np.asarray(dem.targets).astype(np.int32))
