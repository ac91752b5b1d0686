"""Tile heads, rows and spans where the sorted entries are awkward: many
crossings of one tile before its first bin (more than a warp's step, than a
block's), entry counts around the kernel's steps and blocks, rows with gaps
inside and outside the shape, and thousands of one-tile rasters.  Structure
must equal the oracle's, alpha within 1 LSB (the repository's bound)."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _zigzag(n):
    """A raster whose n lines all cross one tile row boundary in one tile, then a wide box."""
    bb = BatchBuilder()
    p = [2.0, 6.5]
    for k in range(n):
        p += [2.0 + 0.003 * (k % 900), 9.5 if k % 2 == 0 else 6.5]
    bb.begin_raster().fill([0] + [1] * n, p, raw=True)
    bb.begin_raster().fill([0, 1, 1, 1], [3.0, 3.0, 700.5, 3.0, 700.5, 60.0, 3.0, 60.0], raw=True)
    return bb.build()


def _combs(n):
    """Rows with many gaps: teeth of a comb, filled between every other pair, and a hole."""
    bb = BatchBuilder()
    for k in range(n):
        bb.begin_raster()
        for q in range(12):
            x = 40.0 * q + 0.37 * k
            bb.fill([0, 1, 1, 1], [x, 1.0, x + 26.0 + q, 1.5, x + 26.0 + q, 43.0 + k % 9, x, 42.0], raw=True)
        bb.fill([0, 1, 1, 1], [0.0, 10.0, 0.0, 30.0, 600.0, 30.0, 600.0, 10.0], raw=True)
    return bb.build()


def _dots(n):
    bb = BatchBuilder()
    for k in range(n):
        bb.begin_raster().fill([0, 1, 1], [k % 97 + 0.2, 1.0, k % 97 + 2.0, 2.0, k % 97 + 0.5, 3.0], raw=True)
    return bb.build()


@pytest.mark.parametrize("name,batch", [(f"zigzag {n}", lambda n=n: _zigzag(n)) for n in (1, 31, 33, 340, 341, 342, 1500, 6000)]
                         + [("combs", lambda: _combs(40)), ("dots", lambda: _dots(5000))])
def test_heads_rows_and_spans_match_oracle(gpu_ctx_chain, name, batch):
    b = batch()
    compare(gpu_ctx_chain.rasterize(b), oracle.run(b, threads=8), b.n_rasters)
