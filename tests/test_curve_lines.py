"""Curves written line by line by neighbouring threads (at least 131,072
commands with at least 8 lines each on average) against the thread that writes
a whole curve: the lines are the same, so the paths' tiles must be those of the
same paths in a smaller call, alpha within 1 LSB (the repository's bound: the
number of tile rows chooses the coverage kernel); and a small call must equal
the oracle's."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _paths(n, seed):
    """Large curves of every kind between moves and lines, some paths left open."""
    rng = np.random.default_rng(seed)
    bb = BatchBuilder()
    for k in range(n):
        p = rng.uniform(0.0, 400.0, 64).astype(np.float32)
        verbs = [[0, 3, 3, 2, 3], [0, 2, 1, 3, 0, 3, 5], [0, 3, 2, 4, 3], [3, 0, 3, 3, 5]][k % 4]
        q, at = [], 0
        for v in verbs:
            m = (2, 2, 4, 6, 5, 0)[v]
            f = [float(x) for x in p[at:at + m]]
            if v == 4:
                f[4] = 0.8
            q += f
            at += m
        bb.begin_raster().fill(verbs, q, raw=True)
    return bb.build()


def test_small_call_matches_oracle(gpu_ctx_chain):
    b = _paths(40, 3)
    compare(gpu_ctx_chain.rasterize(b), oracle.run(b, threads=8), b.n_rasters)


def test_shared_lines_are_the_same_lines(gpu_ctx_chain):
    n = 27_000
    b = _paths(n, 5)
    assert b.n_cmds >= 1 << 17
    whole = gpu_ctx_chain.rasterize(b)
    assert gpu_ctx_chain.stats()["n_lines"] >= 8 * b.n_cmds
    sums = np.add.reduceat(whole["tile_alpha"].sum(1, dtype=np.int64), whole["raster_tile_off"][:-1].astype(np.int64))
    few = _paths(400, 5)
    part = gpu_ctx_chain.rasterize(few)
    t = int(part["raster_tile_off"][-1])
    assert np.array_equal(part["raster_tile_off"], whole["raster_tile_off"][:401])
    assert np.array_equal(part["tile_xy"], whole["tile_xy"][:t])
    assert np.abs(part["tile_alpha"].astype(int) - whole["tile_alpha"][:t].astype(int)).max() <= 1
    assert len(sums) == n and (sums > 0).all()
