"""A wait that gives up after the call has returned.

Compositing returns with its drawing queued.  The test hook
`test_skip_sort_ticket` leaves the first tile of its sort untaken, so the
look-back waits of the other tiles end by their limit (`test_spin_log2`, about a
millisecond): nothing faults or hangs.  The canvas must be as it was, the
context's next rasterizing or compositing call must report the timeout, and the
ones after it must work.
"""
import ctypes

import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300 import DeviceBatch, GpuContext, _lib, workloads

pytestmark = pytest.mark.gpu


def _set(ctx, name, value):
    _lib.check(_lib.load().ochre_gpu_set_tunable(ctx.handle, name.encode(), int(value)), name)


@pytest.mark.parametrize("next_call", ["device", "chain", "host", "composite"])
def test_compositing_that_times_out_is_reported_by_the_next_call(next_call):
    import torch
    b = workloads.glyph_run(n_paths=2000, seed=19, canvas=1024.0)
    exp = oracle.run(b, threads=8)
    L = _lib.load()
    ctx = GpuContext(0, chain_only=next_call == "chain")
    try:
        db = DeviceBatch(b)
        colors = torch.full((b.n_rasters, 4), 77, dtype=torch.uint8, device="cuda:0")
        r = ctx.rasterize_device(db)
        good = torch.full((1024, 1024, 4), 255, dtype=torch.uint8, device="cuda:0")
        ctx.composite(r, b.n_rasters, colors, good)
        torch.cuda.synchronize()

        cv = torch.full((1024, 1024, 4), 255, dtype=torch.uint8, device="cuda:0")
        _set(ctx, "test_spin_log2", 10)
        _set(ctx, "test_skip_sort_ticket", 1)
        ctx.composite(r, b.n_rasters, colors, cv)
        torch.cuda.synchronize()
        assert bool((cv == 255).all())

        q = _lib.Result()
        with pytest.raises(_lib.OchreError) as e:
            if next_call == "host":
                ctx.rasterize(b)
            elif next_call == "composite":
                ctx.composite(r, b.n_rasters, colors, cv)
            else:
                _lib.check(L.ochre_gpu_rasterize_device(ctx.handle, ctypes.byref(db.c), ctypes.byref(q), None))
        assert e.value.status == _lib.E_TIMEOUT

        for _ in range(2):
            r = ctx.rasterize_device(db)
            compare(ctx.device_result_to_numpy(r, b.n_rasters), exp, b.n_rasters)
            cv.fill_(255)
            ctx.composite(r, b.n_rasters, colors, cv)
            torch.cuda.synchronize()
            assert np.array_equal(cv.cpu().numpy(), good.cpu().numpy())
    finally:
        ctx.close()
