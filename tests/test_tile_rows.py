"""Coverage images and their adjoint on canvases whose rows end inside a tile
or lie at odd addresses: an image must be the crop of a larger one (the tile
sums are the same), whatever its width and alignment, and so must dL/dS, which
the gradients show (equal but for the order of their atomic adds: at most some
thousand f32 terms per value, 1e-5 of the gradient's norm)."""
import numpy as np
import pytest

from ochre_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,shift", [(1, 0), (7, 0), (8, 0), (9, 0), (12, 1), (62, 0), (64, 0), (64, 1), (64, 3), (65, 2)])
def test_rows_match_the_crop_of_an_aligned_canvas(gpu_ctx, w, shift):
    import torch
    from ochre_gb300 import DeviceBatch
    b = W.diff_scenes(n_scenes=3, seed=11, size=72.0, max_paths=20, max_seg=24)
    db = DeviceBatch(b)
    big, h = 128, 61
    whole = gpu_ctx.render_coverage(db, big, h).clone()
    room = torch.full((3 * h * w + 8,), -1.0, device="cuda")
    out = room[shift:shift + 3 * h * w].view(3, h, w)
    gpu_ctx.render_coverage(db, w, h, out=out)
    assert torch.equal(out, whole[:, :, :w])
    assert bool((room[:shift] == -1).all()) and bool((room[shift + 3 * h * w:] == -1).all())
    g = torch.Generator(device="cuda").manual_seed(1)
    dl = torch.zeros((3, h, big), device="cuda")
    dl[:, :, :w] = torch.randn((3, h, w), generator=g, device="cuda")
    want = [t.clone() for t in gpu_ctx.fill_backward(db, big, h, dl)]
    dlw = torch.zeros(3 * h * w + 8, device="cuda")
    view = dlw[shift:shift + 3 * h * w].view(3, h, w)
    view.copy_(dl[:, :, :w])
    gpu_ctx.render_coverage(db, w, h, out=out)
    got = gpu_ctx.fill_backward(db, w, h, view)
    for a, e in zip(got, want):
        a, e = a.cpu().numpy().astype(np.float64), e.cpu().numpy().astype(np.float64)
        assert np.linalg.norm(a - e) <= 1e-5 * np.linalg.norm(e)
