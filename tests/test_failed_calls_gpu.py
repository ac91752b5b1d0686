"""A call that fails leaves the context as good as before: the calls after it
give the oracle's output again, on the general chain and on the fused kernel.

Failures are made on the host: a stream that is being captured (refused before
anything is queued, so the capture goes on), and the test hook
`test_fail_scan`, which reports one counted scan as out of memory instead of
launching it.  Nothing here faults, waits out a limit or runs out of memory.
"""
import ctypes

import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300 import DeviceBatch, GpuContext, _lib, workloads

pytestmark = pytest.mark.gpu


def _again(ctx, db, exp):
    """Two calls from device buffers and one from host buffers give the oracle's output."""
    b = db.batch
    for _ in range(2):
        compare(ctx.device_result_to_numpy(ctx.rasterize_device(db), b.n_rasters), exp, b.n_rasters)
    compare(ctx.rasterize(b), exp, b.n_rasters)


def _canvas(ctx, r, b, colors):
    import torch
    cv = torch.full((256, 256, 4), 255, dtype=torch.uint8, device="cuda:0")
    ctx.composite(r, b.n_rasters, colors, cv)
    torch.cuda.synchronize()
    return cv.cpu().numpy()


@pytest.mark.parametrize("chain_only", [False, True], ids=["fused", "chain"])
def test_calls_on_a_capturing_stream_are_refused(chain_only):
    import torch
    b = workloads.glyph_run(n_paths=3000, seed=5, canvas=256.0)
    exp = oracle.run(b, threads=8)
    L = _lib.load()
    ctx = GpuContext(0, chain_only=chain_only)
    try:
        db = DeviceBatch(b)
        _again(ctx, db, exp)
        colors = torch.full((b.n_rasters, 4), 90, dtype=torch.uint8, device="cuda:0")
        r = ctx.rasterize_device(db)
        image = _canvas(ctx, r, b, colors)
        cv = torch.zeros((256, 256, 4), dtype=torch.uint8, device="cuda:0")
        cov = torch.empty((b.n_rasters, 8, 8), device="cuda:0")
        T = r.n_tiles
        buf = {k: torch.empty(n, dtype=torch.uint8, device="cuda:0") for k, n in
               (("tile_xy", 4 * T), ("tile_alpha", 64 * T), ("span_xy", 4 * T), ("span_width", 2 * T),
                ("span_tile", 4 * T), ("raster_tile_off", 4 * (b.n_rasters + 1)),
                ("raster_span_off", 4 * (b.n_rasters + 1)))}
        out = _lib.OutputBuffers(**{k: t.data_ptr() for k, t in buf.items()}, tile_capacity=T, span_capacity=T)
        x = torch.zeros(8, device="cuda:0")
        s = torch.cuda.Stream()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            x += 1.0
            h = s.cuda_stream
            q = _lib.Result()
            st = [L.ochre_gpu_rasterize_device(ctx.handle, ctypes.byref(db.c), ctypes.byref(q), h),
                  L.ochre_gpu_composite(ctx.handle, ctypes.byref(r), b.n_rasters, colors.data_ptr(), 256, 256,
                                        cv.data_ptr(), h),
                  L.ochre_gpu_render_coverage(ctx.handle, ctypes.byref(db.c), 8, 8, cov.data_ptr(), h),
                  L.ochre_gpu_rasterize_noalloc(ctypes.byref(db.c), ctypes.byref(out), h)]
            x += 2.0
        assert st == [_lib.E_CUDA] * 4, st
        g.replay()   # the capture went on around the refused calls
        torch.cuda.synchronize()
        assert x.tolist() == [3.0] * 8 and not cv.any()
        _again(ctx, db, exp)
        assert np.array_equal(_canvas(ctx, ctx.rasterize_device(db), b, colors), image)
    finally:
        ctx.close()


# eager scans of a call: one on the fused kernel; on the chain the commands, line
# counts, line offsets, rasters, tile heads and spans; five more for strokes
@pytest.mark.parametrize("kind,scans", [("fused", 1), ("chain", 6), ("strokes", 11)])
def test_a_scan_that_was_counted_but_not_launched(kind, scans):
    if kind == "strokes":
        b = workloads.stroke_run(n_paths=200, seed=8, canvas=512.0)
    else:
        b = workloads.glyph_run(n_paths=3000, seed=6, canvas=512.0)
    exp = oracle.run(b, threads=8)
    L = _lib.load()
    ctx = GpuContext(0, chain_only=kind != "fused")
    try:
        db = DeviceBatch(b)
        _again(ctx, db, exp)
        r = _lib.Result()
        failed = 0
        for k in range(1, scans + 1):
            _lib.check(L.ochre_gpu_set_tunable(ctx.handle, b"test_fail_scan", k))
            st = L.ochre_gpu_rasterize_device(ctx.handle, ctypes.byref(db.c), ctypes.byref(r), None)
            _lib.check(L.ochre_gpu_set_tunable(ctx.handle, b"test_fail_scan", 0))
            failed += st == _lib.E_NOMEM
            _again(ctx, db, exp)
        assert failed == scans, (failed, scans)
    finally:
        ctx.close()


def test_compositing_after_a_failed_scan():
    import torch
    b = workloads.glyph_run(n_paths=500, seed=7, canvas=256.0)
    L = _lib.load()
    ctx = GpuContext(0)
    try:
        db = DeviceBatch(b)
        colors = torch.full((b.n_rasters, 4), 120, dtype=torch.uint8, device="cuda:0")
        r = ctx.rasterize_device(db)
        image = _canvas(ctx, r, b, colors)
        _lib.check(L.ochre_gpu_set_tunable(ctx.handle, b"test_fail_scan", 1))
        with pytest.raises(_lib.OchreError) as e:
            _canvas(ctx, r, b, colors)
        assert e.value.status == _lib.E_NOMEM
        assert np.array_equal(_canvas(ctx, r, b, colors), image)
    finally:
        ctx.close()
