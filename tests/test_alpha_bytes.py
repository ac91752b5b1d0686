"""Alpha bytes where a sum lies on, just under and far past a step of 1/256:
boxes of height k/256 and the float below it, of both windings, single and
stacked past 255/256.  A byte is a function of its cell's sum alone, so it must
be min(floor(|sum| * 256), 255) of the coverage that the same run returns,
exactly (the product by 256 is exact), on the fused path and on the general one."""
import numpy as np
import pytest

from ochre_gb300 import GpuContext
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _boxes():
    bb = BatchBuilder()
    for k in range(1, 257):
        for h in (k / 256.0, float(np.nextafter(np.float32(k / 256.0), np.float32(0)))):
            for p in ([0.0, 0.0, 16.0, 0.0, 16.0, h, 0.0, h], [0.0, 0.0, 0.0, h, 16.0, h, 16.0, 0.0]):
                bb.begin_raster().fill([0, 1, 1, 1], p, raw=True)
    for n in (2, 5):   # the same box n times: past the byte's range
        bb.begin_raster()
        for _ in range(n):
            bb.fill([0, 1, 1, 1], [0.0, 0.0, 16.0, 0.0, 16.0, 0.75, 0.0, 0.75], raw=True)
    return bb.build()


def _check(out):
    want = np.minimum(np.floor(np.abs(out["tile_cov"].astype(np.float64)) * 256.0), 255).astype(np.uint8)
    assert np.array_equal(out["tile_alpha"], want)
    assert len(np.unique(want)) == 256


@pytest.mark.parametrize("chain", [False, True])
def test_bytes_on_the_steps(chain):
    ctx = GpuContext(0, want_cov=True, chain_only=chain)
    _check(ctx.rasterize(_boxes()))
