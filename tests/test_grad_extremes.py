"""The backward on inputs far from any picture: what no pixel sees has gradient
0 however far away it lies, and a gradient past the largest number is infinite."""
import numpy as np
import pytest

from ochre_gb300 import DeviceBatch, GpuContext
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _gradients(batch, w, h, dl):
    import torch
    ctx = GpuContext(0)
    try:
        db = DeviceBatch(batch)
        ctx.render_coverage(db, w, h)
        p, x = ctx.fill_backward(db, w, h, torch.as_tensor(dl, device="cuda:0"))
        return p.cpu().numpy()[:len(batch.pts)], x.cpu().numpy()
    finally:
        ctx.close()


_SHAPE = [3.3, 4.1, 27.6, 6.2, 20.4, 25.9]


@pytest.mark.parametrize("far", [[2.5e38, 5.0, 2.5e38, 21.0], [-2.5e38, 40.5, -2.5e38, 60.0],
                                 [3.0e38, -9.0, 3.0e38, 70.5]])
def test_far_lines_have_no_gradient(far):
    """A line at coordinates whose sums overflow, right of the canvas or off its rows, and back."""
    dl = np.random.default_rng(3).normal(size=(1, 32, 32)).astype(np.float32)
    near, _ = _gradients(BatchBuilder().begin_raster().fill([0, 1, 1], _SHAPE, raw=True).build(), 32, 32, dl)
    b = BatchBuilder().begin_raster().fill([0, 1, 1, 0, 1], _SHAPE + far, raw=True).build()
    p, _ = _gradients(b, 32, 32, dl)
    assert np.count_nonzero(near) == 6
    assert np.array_equal(p[6:], np.zeros(4, np.float32)), p
    # (the same terms, their atomic adds in any order)
    assert np.allclose(p[:6], near, rtol=1e-5, atol=1e-5 * np.abs(near).max()), (p, near)


def test_products_past_the_largest_number_are_infinite():
    """One pixel's gradient on a line, where the line crosses from one pixel column
    to the next: gradient * height and gradient * width overflow, each with one
    sign, and no infinity meets another or a 0."""
    w, h = 80, 320
    b = BatchBuilder().begin_raster().fill([0, 1, 1], [2.5, 2.5, 66.5, 302.5, 70.25, 150.5], raw=True).build()
    # the line goes from column 18 to column 19 at y = 79.84
    dl = np.zeros((1, h, w), np.float32)
    dl[0, 79, 18] = 1e38
    p, _ = _gradients(b, w, h, dl)
    assert not np.isnan(p).any(), p
    assert np.isinf(p[:2]).all() and np.isfinite(p[2:]).all(), p
