"""Batches whose lines are mostly long: one thread walks each of them then, as it
does the short ones.  Outputs as the oracle's on both sides of the rule (an
eighth of the lines long, and 32,768 of them), and the emission's time against
a context that walks every line by one thread."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300 import DeviceBatch, GpuContext, autotune
from ochre_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _polygons(n, lines, extent, short=0):
    """n rasters, each a closed polygon of `lines` random lines within `extent`
    pixels, and after them `short` lines a few pixels long."""
    rng = np.random.default_rng(17)
    x = rng.uniform(0.0, extent, (n, lines, 2))
    tail = x[:, -1:, :] + np.cumsum(rng.uniform(-2.0, 2.0, (n, short, 2)), axis=1)
    pts = np.concatenate([x, tail], axis=1).astype(np.float32)
    k = lines + short
    verbs = np.tile(np.r_[0, np.ones(k - 1)].astype(np.uint8), n)
    xf = np.tile(np.array([1, 0, 0, 1, 0, 0], np.float32), (n, 1))
    return Batch(verbs, pts.reshape(-1), (np.arange(n + 1) * k).astype(np.uint32), xf, None, None, n)


# long lines: few; under and over 32,768; many, but under and over an eighth
@pytest.mark.parametrize("n,lines,short", [(40, 30, 0), (350, 100, 0), (400, 100, 0), (500, 100, 900), (500, 100, 500)])
def test_long_lines_match_oracle(n, lines, short):
    b = _polygons(n, lines, 400.0, short)
    exp = oracle.run(b, threads=16)
    ctx = GpuContext(0, chain_only=True)
    try:
        db = DeviceBatch(b)
        compare(ctx.device_result_to_numpy(ctx.rasterize_device(db), n), exp, n)
        g = ctx.graph(db)
        compare(g.rasterize(), exp, n)
        g.close()
    finally:
        ctx.close()


def test_many_long_lines_take_no_longer_than_by_one_thread_each():
    """1.2 M lines, two thirds of them of 97 to 384 cells (within a tenth: times)."""
    b = _polygons(12_000, 100, 200.0)
    ms = []
    for cells in (96, 0):
        ctx = GpuContext(0, chain_only=True, profile=True)
        try:
            autotune.apply(ctx, {"chain_long_cells": cells})
            db = DeviceBatch(b)
            best = 1e9
            for _ in range(6):
                ctx.rasterize_device(db)
                t = dict(ctx.timings())
                best = min(best, max(t["dda_emit"], t.get("dda_emit_long", 0.0)))
            ms.append(best)
        finally:
            ctx.close()
    assert ms[0] < 1.1 * ms[1], ms
