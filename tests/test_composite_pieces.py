"""The compositing kernel at its edges: division by 255, more pieces on a
screen tile than a warp takes at once, canvases that end inside a tile, keys
of 32 and 64 bits, fewer rasters than the result holds, and an alpha array at
an odd address.  Bytes must equal the oracle's."""
from fractions import Fraction

import numpy as np
import pytest

import oracle
from ochre_gb300 import _lib, workloads as W
from ochre_gb300.batch import BatchBuilder


def _round_f32(x: Fraction) -> Fraction:
    if x == 0:
        return Fraction(0)
    e = -30
    while Fraction(2) ** (e + 1) <= abs(x):
        e += 1
    q = Fraction(2) ** (e - 23)
    return round(x / q) * q   # round half to even


def test_division_by_255_with_one_correction_is_correctly_rounded():
    rcp = _round_f32(Fraction(1, 255))
    assert float(rcp) == float.fromhex("0x1.010102p-8")
    for x in range(256):
        q = _round_f32(x * rcp)
        r = _round_f32(x - 255 * q)
        assert _round_f32(r * rcp + q) == _round_f32(Fraction(x, 255)), x


def _stack(n):
    """n translucent shapes over the same few screen tiles."""
    bb = BatchBuilder()
    for k in range(n):
        bb.begin_raster().fill([0, 1, 1, 1, 5], [2.0 + k % 5, 3.0, 70.5, 5.0 + k % 7, 50.0, 71.0, 3.0, 60.0 - k % 11])
    return bb.build()


@pytest.mark.gpu
@pytest.mark.parametrize("name,batch,w,h,draw,odd", [
    ("31 pieces", lambda: _stack(31), 75, 73, None, False),
    ("32 pieces", lambda: _stack(32), 75, 73, None, False),
    ("33 pieces", lambda: _stack(33), 75, 73, None, True),
    ("100 pieces", lambda: _stack(100), 80, 80, None, False),
    ("narrow canvas", lambda: _stack(40), 1, 64, None, False),
    ("some rasters", lambda: _stack(64), 75, 73, 32, False),
    ("64-bit keys", lambda: W.glyph_run(n_paths=4200, seed=9, canvas=8192.0), 8192, 8192, None, False),
])
def test_composite_edges_match_oracle(name, batch, w, h, draw, odd):
    import torch
    from ochre_gb300 import DeviceBatch, GpuContext
    b = batch()
    n = b.n_rasters if draw is None else draw
    rng = np.random.default_rng(3)
    colors = rng.integers(0, 256, size=(b.n_rasters, 4), dtype=np.uint8)
    canvas = rng.integers(0, 256, size=(h, w, 4), dtype=np.uint8)
    ctx = GpuContext(0)
    try:
        stream = torch.cuda.current_stream().cuda_stream
        r = ctx.rasterize_device(DeviceBatch(b, 0), stream)
        res = ctx.device_result_to_numpy(r, b.n_rasters)
        if odd:
            alpha = torch.zeros(r.n_tiles * 64 + 1, dtype=torch.uint8, device="cuda:0")
            alpha[1:] = torch.as_tensor(res["tile_alpha"].reshape(-1), device="cuda:0")
            assert alpha.data_ptr() % 2 == 0
            moved = _lib.Result.from_buffer_copy(r)
            moved.tile_alpha = alpha.data_ptr() + 1
            r = moved
        cv = torch.as_tensor(canvas, device="cuda:0").clone()
        ctx.composite(r, n, torch.as_tensor(colors, device="cuda:0"), cv)
        got = cv.cpu().numpy()
    finally:
        ctx.close()
    if draw is not None:
        t, s = int(res["raster_tile_off"][n]), int(res["raster_span_off"][n])
        for k, m in (("tile_xy", t), ("tile_alpha", t), ("span_xy", s), ("span_w", s), ("span_tile", s),
                     ("raster_tile_off", n + 1), ("raster_span_off", n + 1)):
            res[k] = res[k][:m]
    ref = oracle.composite(res, n, colors[:n], w, h, canvas)
    assert np.array_equal(got, ref), (name, int((got != ref).any(axis=2).sum()))
