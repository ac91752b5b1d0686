"""Many rasters of few sort entries: on both sides of the rule that chooses between
a block per raster and the device-wide passes (entries + 2^20 >= 96 rasters) the
outputs are the oracle's, and the sort takes no longer than by the passes alone
(11-bit digits keep the chain to them; a third is for their other widths)."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300 import DeviceBatch, GpuContext, autotune
from ochre_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _dots(n, lines, extent):
    """n rasters, each a closed polygon of `lines` random lines within `extent` pixels."""
    pts = np.random.default_rng(23).uniform(0.0, extent, (n, lines, 2)).astype(np.float32)
    verbs = np.tile(np.r_[0, np.ones(lines - 1)].astype(np.uint8), n)
    xf = np.tile(np.array([1, 0, 0, 1, 0, 0], np.float32), (n, 1))
    return Batch(verbs, pts.reshape(-1), (np.arange(n + 1) * lines).astype(np.uint32), xf, None, None, n)


@pytest.mark.parametrize("n,lines,extent,passes", [(3000, 3, 6.0, 1), (11_000, 3, 6.0, 1), (12_000, 3, 6.0, 2),
                                                   (20_000, 8, 30.0, 3), (20_000, 10, 60.0, 1)])
def test_small_rasters_match_oracle(n, lines, extent, passes):
    b = _dots(n, lines, extent)
    exp = oracle.run(b, threads=16)
    ctx = GpuContext(0, chain_only=True)
    try:
        compare(ctx.device_result_to_numpy(ctx.rasterize_device(DeviceBatch(b)), n), exp, n)
        s = ctx.stats()
        assert (s["sort_passes"] == 1) == (s["n_entries"] + (1 << 20) >= 96 * n) == (passes == 1), s
    finally:
        ctx.close()


def test_sort_of_a_million_tiny_rasters():
    b = _dots(1_000_000, 3, 6.0)
    us = []
    for digit_bits in (8, 11):
        ctx = GpuContext(0, chain_only=True, profile=True)
        try:
            autotune.apply(ctx, {"sort_digit_bits": digit_bits})
            db = DeviceBatch(b)
            best = 1e9
            for _ in range(5):
                ctx.rasterize_device(db)
                best = min(best, 1000 * sum(ms for name, ms in ctx.timings() if name.startswith("sort")))
            us.append(best)
        finally:
            ctx.close()
    assert us[0] < 1.34 * us[1], us
