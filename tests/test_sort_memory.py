"""Look-back words of the radix sort: passes have words of their own only while
those take little memory; a long sort's passes share one set.  Both give the
same order (equal outputs: the sort is stable and everything after it is the same)."""
import numpy as np
import pytest

from ochre_gb300 import DeviceBatch, GpuContext, autotune, workloads

pytestmark = pytest.mark.gpu


def test_long_sorts_share_their_look_back_words():
    import torch
    b = workloads.uneven_mix(n_paths=2000, seed=21)
    ctx = GpuContext(0, chain_only=True)
    try:
        db = DeviceBatch(b)
        got = ctx.device_result_to_numpy(ctx.rasterize_device(db), b.n_rasters)
        st = ctx.stats()
        # a tile of 3,840 entries has 256 or 2,048 words a pass
        tiles = (st["n_entries"] + 3839) // 3840
        assert st["sort_passes"] > 1 and (st["sort_passes"] - 1) * tiles * 256 * 4 < 64 << 20
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        autotune.apply(ctx, {"sort_digit_bits": 11})
        wide = ctx.device_result_to_numpy(ctx.rasterize_device(db), b.n_rasters)
        assert (ctx.stats()["sort_passes"] - 1) * tiles * 2048 * 4 > 64 << 20
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()
    # one pass's words, in a buffer of up to twice their size
    assert used <= 2 * tiles * 2048 * 4, used
    for k in got:
        assert np.array_equal(got[k], wide[k]), k
