"""Coverage kernels over tile rows of every length around their chunks (4, 8,
16 tiles) and metadata windows (32, 64), starting at every place in a window,
with few and with many entries a tile, in both forms.  Structure must equal the
oracle's, alpha within 1 LSB (the repository's bound)."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300 import GpuContext, autotune
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _rows():
    bb = BatchBuilder()
    for n in list(range(1, 36)) + [47, 48, 49, 63, 64, 65, 66, 95, 97, 130, 200]:
        bb.begin_raster()
        for r in range(1 + n % 3):
            y = 8.0 * r + 0.2
            bb.fill([0, 1, 1, 1], [0.4, y + 1.1, 8.0 * n - 0.6, y + 2.3, 8.0 * n - 0.6, y + 6.4, 0.4, y + 4.9], raw=True)
    return bb.build()


def _dense():
    """Tiles with 1 to some hundred bins, in rows of a few to 80 tiles."""
    rng = np.random.default_rng(9)
    bb = BatchBuilder()
    for k, n in enumerate((3, 8, 9, 17, 33, 80)):
        bb.begin_raster()
        m = 40 * n
        p = np.stack([rng.uniform(0, 8.0 * n, m), rng.uniform(0, 20.0, m)], 1).astype(np.float32)
        q = p + rng.uniform(-3, 3, (m, 2)).astype(np.float32)
        z = p + rng.uniform(-3, 3, (m, 2)).astype(np.float32)
        for i in range(m):
            bb.fill([0, 1, 1], [*p[i], *q[i], *z[i]], raw=True)
    return bb.build()


@pytest.mark.parametrize("form", [1, 2])
@pytest.mark.parametrize("tiles", [4, 8, 16])
@pytest.mark.parametrize("name", ["rows", "dense"])
def test_rows_match_oracle(name, tiles, form):
    ctx = GpuContext(0, chain_only=True)
    autotune.apply(ctx, {"chain_coverage_form": form, "chain_tiles_per_warp": tiles})
    b = _rows() if name == "rows" else _dense()
    compare(ctx.rasterize(b), oracle.run(b, threads=8), b.n_rasters)
