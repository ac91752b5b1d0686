"""The fused kernel's rasters where its phases have edges: touched tiles around
a chunk (8, 16, 32) and the raster's limit (128), rows cut by a chunk,
crossings in every remainder of four, empty rasters between others, lines at
the ends of the i16 range (fused or handed to the general chain), curves of
every kind, and fewer, as many and more rasters than the kernel has blocks.
Structure must equal the oracle's, alpha within 1 LSB (the repository's bound)."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300 import GpuContext, autotune
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _strip(bb, tiles, rows, y0=0.0):
    """A zigzag that touches `tiles` tiles of each of `rows` tile rows, half covered."""
    bb.begin_raster()
    for r in range(rows):
        y = y0 + 8.0 * r
        bb.fill([0, 1, 1, 1], [0.5, y + 1.25, 8.0 * tiles - 0.5, y + 2.5, 8.0 * tiles - 0.5, y + 6.5, 0.5, y + 5.0], raw=True)


def _chunks():
    bb = BatchBuilder()
    for n in (1, 2, 7, 8, 9, 15, 16, 17, 23, 24, 25, 29, 30):
        _strip(bb, n, 1)
        bb.begin_raster()                       # an empty raster between
        _strip(bb, n, 2, 0.3)
    for rows in (3, 4, 5, 8, 15, 16):           # up to 128 touched tiles
        _strip(bb, 8, rows)
    return bb.build()


def _crossings():
    bb = BatchBuilder()
    for n in range(1, 14):
        p = [2.0, 6.5]
        for k in range(n):
            p += [2.0 + 0.7 * k, 9.5 if k % 2 == 0 else 6.5]
        bb.begin_raster().fill([0] + [1] * n, p, raw=True)
        bb.begin_raster()
        for k in range(min(n, 7)):              # spans between nested boxes
            bb.fill([0, 1, 1, 1], [1.0 + 24 * k, 1.0, 20.0 + 24 * k, 1.5, 20.0 + 24 * k, 60.0, 1.0 + 24 * k, 59.0], raw=True)
    return bb.build()


def _limits():
    bb = BatchBuilder()
    for x in (32740.0, 32759.5, 32767.25, 32768.0, 32790.0, -32768.0, -32770.5, -32800.0):
        for y in (3.0, x):
            bb.begin_raster().fill([0, 1, 1, 1], [x, y, x - 9.5, y + 4.0, x + 11.0, y + 13.0, x + 2.0, y - 6.0], raw=True)
    return bb.build()


def _curves(n):
    rng = np.random.default_rng(5)
    bb = BatchBuilder()
    for k in range(n):
        bb.begin_raster()
        p = rng.uniform(0.0, 40.0, 24).astype(np.float32)
        if k % 3 == 0:
            bb.fill([0, 2, 3, 1, 5], p[:14], raw=True)
        elif k % 3 == 1:
            bb.fill([0, 1, 2, 1], p[:10], raw=True)
        else:
            bb.fill([0, 4, 1, 4], [*p[:6], 0.7, *p[7:9], *p[9:13], 1.4], raw=True)
    return bb.build()


@pytest.mark.parametrize("threads,chunk", [(64, 8), (64, 16), (64, 32), (96, 16), (128, 32)])
@pytest.mark.parametrize("name", ["chunks", "crossings", "limits"])
def test_edges_match_oracle(name, threads, chunk):
    ctx = GpuContext(0)
    autotune.apply(ctx, {"fused_threads": threads, "fused_chunk": chunk})
    b = {"chunks": _chunks, "crossings": _crossings, "limits": _limits}[name]()
    compare(ctx.rasterize(b), oracle.run(b, threads=8), b.n_rasters)
    if name != "limits":
        assert ctx.stats()["fused"] == 1


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 2127, 2128, 2129, 4300, 9001])
def test_raster_counts_match_oracle(gpu_ctx, n):
    b = _curves(n)
    compare(gpu_ctx.rasterize(b), oracle.run(b, threads=8), b.n_rasters)
    assert gpu_ctx.stats()["fused"] == 1
