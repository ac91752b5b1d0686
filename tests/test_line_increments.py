"""Increments of lines of every length and start within a 32-byte sector, in
both directions, and of lines that begin past the i16 range of cells (whose
first steps lie below parameter 0).  Structure must equal the oracle's, alpha
within 1 LSB (the repository's bound)."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _lengths():
    """Saw teeth whose edges cross 1 to 21 cells, in an order that meets every start modulo 4."""
    bb = BatchBuilder()
    rng = np.random.default_rng(1)
    for k in range(60):
        bb.begin_raster()
        p, x, y = [0.3, 0.4], 0.3, 0.4
        n = int(rng.integers(3, 40))
        for q in range(n):
            c = int(rng.integers(0, 22))
            dx = int(rng.integers(0, c + 1))
            x += dx * (1 if rng.random() < 0.6 else -1)
            y += (c - dx) * (1 if rng.random() < 0.6 else -1)
            p += [x, y]
        bb.fill([0] + [1] * n, p, raw=True)
    return bb.build()


def _past_the_range():
    bb = BatchBuilder()
    for d in (0.5, 1.0, 7.75, 40.0):
        for x0, y0 in ((32767.0, 5.0), (32767.0, 32767.0), (-32768.0, 5.0), (-32768.0, -32768.0), (5.0, -32768.0)):
            sx, sy = np.sign(x0), (np.sign(y0) if abs(y0) > 100 else 0.0)
            a = [x0 + sx * d, y0 + sy * d]
            p = a + [x0 - sx * 9.25, y0 + 3.5] + [x0 + sx * (d + 3.0), y0 + sy * (d + 2.5)] + [x0 - sx * 4.0, y0 - 6.0]
            bb.begin_raster().fill([0, 1, 1, 1], p, raw=True)
    return bb.build()


@pytest.mark.parametrize("name", ["lengths", "past the range"])
def test_lines_match_oracle(gpu_ctx_chain, name):
    b = _lengths() if name == "lengths" else _past_the_range()
    compare(gpu_ctx_chain.rasterize(b), oracle.run(b, threads=8), b.n_rasters)
