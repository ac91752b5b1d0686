"""A fused shape that is not built (96 threads with chunks of 32 tiles) is refused
whatever the batch, also one with more commands than its rasters could take on
the fused kernel; on a context that uses the chain alone it plays no part."""
import ctypes

import pytest

import oracle
from compare import compare
from ochre_gb300 import DeviceBatch, GpuContext, _lib, autotune, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,batch", [("glyphs", lambda: workloads.glyph_run(n_paths=50, seed=4)),
                                        ("long paths", lambda: workloads.uneven_mix(n_paths=3, seed=4, median=500.0,
                                                                                    sigma=0.0, canvas=700.0))])
def test_unbuilt_shape_is_refused(name, batch):
    b = batch()
    assert (b.n_cmds > 96 * b.n_rasters) == (name == "long paths")
    exp = oracle.run(b, threads=8)
    L = _lib.load()
    ctx = GpuContext(0)
    try:
        db = DeviceBatch(b)
        autotune.apply(ctx, {"fused_threads": 96, "fused_chunk": 32})
        r = _lib.Result()
        for _ in range(2):
            assert L.ochre_gpu_rasterize_device(ctx.handle, ctypes.byref(db.c), ctypes.byref(r), None) == _lib.E_INVALID
        with pytest.raises(_lib.OchreError) as e:
            ctx.rasterize(b)
        assert e.value.status == _lib.E_INVALID
        ctx.set_chain_only(True)
        compare(ctx.device_result_to_numpy(ctx.rasterize_device(db), b.n_rasters), exp, b.n_rasters)
        ctx.set_chain_only(False)
        autotune.apply(ctx, {"fused_threads": 96, "fused_chunk": 16})
        compare(ctx.device_result_to_numpy(ctx.rasterize_device(db), b.n_rasters), exp, b.n_rasters)
    finally:
        ctx.close()
