"""The entry sort by one block per raster at its limits: entry counts around
each block size (and past the largest, where the device-wide sort runs), key
spaces of 1 to 19 bits and past that, rasters without increments between the
others, and few or many rasters.  Structure must equal the oracle's, alpha
within 1 LSB (the repository's bound)."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _dots(bb, n, tiles_x, tiles_y, rng):
    """A raster of n two-line contours, each inside one pixel: 2 n entries."""
    bb.begin_raster()
    if n == 0:
        return
    cell = np.stack([rng.integers(0, 8 * tiles_x, n), rng.integers(0, 8 * tiles_y, n)], axis=1)
    cell[0] = 0
    cell[-1] = (8 * tiles_x - 1, 8 * tiles_y - 1)
    a = cell + rng.uniform(0.1, 0.9, (n, 2))
    b = cell + rng.uniform(0.1, 0.9, (n, 2))
    bb.fill(np.tile(np.array([0, 1], np.uint8), n), np.concatenate([a, b], axis=1).astype(np.float32).reshape(-1), raw=True)


@pytest.mark.parametrize("sizes,tiles", [
    ([1, 0, 511, 0, 0, 512, 513], (16, 16)),            # the small block's limit
    ([2047, 2048, 2049, 3, 0], (1, 1)),                 # the middle block's, one tile
    ([4095, 4096, 0, 700], (40, 7)),                    # the large block's
    ([4096, 4097, 0, 5], (40, 7)),                      # past it
    ([300, 0, 900], (512, 512)),                        # 19 key bits
    ([300, 0, 900], (513, 512)),                        # past them
    ([(k * 37) % 600 for k in range(1500)], (9, 11)),   # many rasters, two sizes
    ([5000 if k == 700 else (k * 37) % 60 for k in range(1500)], (9, 11)),
])
def test_block_sizes_match_oracle(gpu_ctx_chain, sizes, tiles):
    rng = np.random.default_rng(len(sizes) + tiles[0])
    bb = BatchBuilder()
    for n in sizes:
        _dots(bb, n, *tiles, rng)
    b = bb.build()
    compare(gpu_ctx_chain.rasterize(b), oracle.run(b, threads=8), b.n_rasters)
