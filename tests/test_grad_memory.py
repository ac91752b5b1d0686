"""The backward's per-pixel memory: one image of (dL/dS, suffix sum) pairs, 8
bytes a pixel, filled in place row by row."""
import numpy as np
import pytest

from ochre_gb300 import DeviceBatch, GpuContext
from ochre_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_backward_keeps_eight_bytes_a_pixel():
    import torch
    w = h = 4096
    b = W.diff_union(n_paths=4, seed=3)
    ctx = GpuContext(0)
    try:
        db = DeviceBatch(b)
        dl = ctx.render_coverage(db, w, h)
        p = torch.empty(len(b.pts), device="cuda:0")
        x = torch.empty((b.n_fills, 6), device="cuda:0")
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ctx.fill_backward(db, w, h, dl, p, x)
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()
    # (and what a few thousand lines, points and rows take, allocated in whole 2 MB pages)
    assert used <= 8 * w * h + (16 << 20), used


# rows that end before, at and past the 32 values of a step
@pytest.mark.parametrize("w", [31, 32, 33, 63, 95, 96, 97, 129])
def test_rows_in_place_match_the_crop_of_a_wider_canvas(gpu_ctx, w):
    """As in test_tile_rows.py: the gradients of a crop (the same terms, their atomic
    adds in any order: 1e-5 of the gradient's norm)."""
    import torch
    b = W.diff_scenes(n_scenes=2, seed=12, size=140.0, max_paths=20, max_seg=24)
    db = DeviceBatch(b)
    big, h = 256, 77
    g = torch.Generator(device="cuda").manual_seed(2)
    dl = torch.zeros((2, h, big), device="cuda")
    dl[:, :, :w] = torch.randn((2, h, w), generator=g, device="cuda")
    want = [t.clone() for t in gpu_ctx.fill_backward(db, big, h, dl)]
    got = gpu_ctx.fill_backward(db, w, h, dl[:, :, :w].contiguous())
    for a, e in zip(got, want):
        a, e = a.cpu().numpy().astype(np.float64), e.cpu().numpy().astype(np.float64)
        assert np.linalg.norm(e) > 0 and np.linalg.norm(a - e) <= 1e-5 * np.linalg.norm(e)
