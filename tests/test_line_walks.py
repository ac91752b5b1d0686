"""Line counts without a walk and the long lines' walk by groups of lanes, on
lines where the walk's ties, boundaries and limits lie: ends on pixel and tile
boundaries, exact diagonals, axis-parallel lines, one cell, both sides of the
16- and 32-cell rounds, thousands of cells, and the i16 limits.  Structure
must equal the oracle's, alpha within 1 LSB (the repository's bound)."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _lines(n, reach, seed):
    """n triangles of raw lines of about `reach` px, many of their ends on boundaries."""
    rng = np.random.default_rng(seed)
    bb = BatchBuilder()
    for k in range(n):
        o = rng.uniform(-reach, reach, 2)
        p = o + rng.uniform(-reach, reach, (3, 2))
        kind = k % 8
        if kind == 1:
            p = np.floor(p)
        elif kind == 2:
            p = np.floor(p / 8.0) * 8.0
        elif kind == 3:
            p[1] = p[0] + (p[1, 0] - p[0, 0])          # an exact diagonal
        elif kind == 4:
            p[1, 1] = p[0, 1]                          # horizontal, then vertical
            p[2, 0] = p[1, 0]
        elif kind == 5:
            p = np.floor(p * 4.0) / 4.0
        elif kind == 6:
            p[1] = p[0] + rng.uniform(-0.9, 0.9, 2)    # a short line
        p = p.astype(np.float32)
        bb.begin_raster().fill([0, 1, 1], p.reshape(-1), raw=True)
    return bb.build()


def _limits():
    bb = BatchBuilder()
    for p in ([32700.5, 10.25, 33100.0, 90.5, 32500.0, 77.0], [5.0, 32750.0, 60.5, 33000.0, 70.0, 32600.25],
              [-32760.0, 3.0, -33000.0, 50.0, -32700.0, 60.0]):
        bb.begin_raster().fill([0, 1, 1], p, raw=True)
    return bb.build()


@pytest.mark.parametrize("long_cells", [0, 16, 96])
@pytest.mark.parametrize("name,batch", [
    ("few short", lambda: _lines(24, 20, 1)),
    ("few long", lambda: _lines(40, 900, 2)),            # a warp per line
    ("many", lambda: _lines(3000, 120, 3)),              # more long lines than warps: four share one
    ("limits", _limits),
])
def test_counts_and_walks_match_oracle(gpu_ctx_chain, name, batch, long_cells):
    from ochre_gb300 import autotune
    b = batch()
    ref = oracle.run(b, threads=8)
    old = autotune.get(gpu_ctx_chain, "chain_long_cells")
    try:
        autotune.apply(gpu_ctx_chain, {"chain_long_cells": long_cells})
        got = gpu_ctx_chain.rasterize(b)
    finally:
        autotune.apply(gpu_ctx_chain, {"chain_long_cells": old})
    compare(got, ref, b.n_rasters)
