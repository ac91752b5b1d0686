"""Crossings of tiles without bins.

A line from the upper left that ends exactly on a tile's corner snaps there and
leaves its row crossing in a tile it has no cell in (the lines below never enter
the tile at (8, 0), which keeps their crossings and no bin).  However many such
crossings lie between two tiles, the tile heads must come out as the oracle's,
and no wait of the run may outlast its limit while they are passed over.
"""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300 import DeviceBatch, GpuContext, _lib, autotune
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _corner(n):
    """n lines (5,5) -> (8,8) -> (5,5) .., a box beside them, then a wide raster and a small one."""
    bb = BatchBuilder()
    p = np.empty((n + 1, 2), np.float32)
    p[0::2], p[1::2] = 5.0, 8.0
    bb.begin_raster()
    bb.fill(np.r_[0, np.ones(n, int)], p, raw=True)
    bb.fill([0, 1, 1, 1], [30.0, 2.0, 61.5, 2.0, 61.5, 22.0, 30.0, 22.0], raw=True)
    bb.begin_raster().fill([0, 1, 1, 1], [3.0, 3.0, 700.5, 3.0, 700.5, 60.0, 3.0, 60.0], raw=True)
    bb.begin_raster().fill([0, 1, 1], [1.2, 1.0, 6.0, 2.0, 3.5, 5.0], raw=True)
    return bb.build()


# crossings: n / 2; around a warp's look at the entries before it, a warp's
# entries (128 and 512) and a block's (1,024 and 4,096)
@pytest.mark.parametrize("n", [2, 62, 64, 66, 254, 258, 1022, 1030, 2046, 2050, 8190, 8200, 60_000])
def test_corner_crossings_match_oracle(gpu_ctx_chain, n):
    b = _corner(n)
    exp = oracle.run(b, threads=8)
    assert [8, 0] not in exp["tile_xy"][:exp["raster_tile_off"][1]].tolist()
    compare(gpu_ctx_chain.rasterize(b), exp, b.n_rasters)


def test_many_corner_crossings_outlast_no_wait():
    """Two million lines, waits of at most 2^12 polls (a few milliseconds); the
    row form of the coverage kernel has no waits of its own."""
    b = _corner(2_000_000)
    exp = oracle.run(b, threads=8)
    ctx = GpuContext(0, chain_only=True)
    try:
        autotune.apply(ctx, {"chain_coverage_form": 2})
        db = DeviceBatch(b)
        ctx.rasterize_device(db)   # (buffers grow)
        _lib.check(_lib.load().ochre_gpu_set_tunable(ctx.handle, b"test_spin_log2", 12))
        compare(ctx.device_result_to_numpy(ctx.rasterize_device(db), b.n_rasters), exp, b.n_rasters)
    finally:
        ctx.close()
