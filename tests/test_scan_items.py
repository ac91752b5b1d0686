"""Command counts around a scan thread's items (2 below 65,537 commands, 8
above) and blocks, with the command bytes at every alignment: structure must
equal the oracle's, alpha within 1 LSB (the repository's bound), on the fused
path and on the general one."""
import numpy as np
import pytest

import oracle
from compare import compare
from ochre_gb300 import GpuContext
from ochre_gb300.batch import BatchBuilder

pytestmark = pytest.mark.gpu


def _commands(n):
    """n commands in all: small closed shapes of 4 to 12, lines and curves."""
    rng = np.random.default_rng(n)
    bb = BatchBuilder()
    left = n
    while left > 0:
        k = left if left < 16 else int(rng.integers(4, 13))
        left -= k
        v = [0] + [int(x) for x in rng.choice([1, 1, 2, 3], k - 1)]
        p = rng.uniform(0.0, 30.0, sum((2, 2, 4, 6)[x] for x in v)).astype(np.float32)
        bb.begin_raster().fill(v, p, raw=True)
    return bb.build()


@pytest.mark.parametrize("chain", [False, True])
@pytest.mark.parametrize("n,shift", [(1, 0), (2, 1), (7, 0), (8, 0), (9, 3), (511, 0), (513, 7), (2049, 0), (65536, 0),
                                     (65537, 0), (65537, 4), (67583, 1), (67585, 8)])
def test_counts_and_alignments_match_oracle(n, shift, chain):
    import torch
    from ochre_gb300 import DeviceBatch
    b = _commands(n)
    ctx = GpuContext(0, chain_only=chain)
    db = DeviceBatch(b)
    room = torch.zeros(n + 16, dtype=torch.uint8, device="cuda")
    room[shift:shift + n] = db.verbs[:n]
    db.c.verbs = room.data_ptr() + shift
    res = ctx.rasterize_device(db)
    compare(ctx.device_result_to_numpy(res, b.n_rasters), oracle.run(b, threads=8), b.n_rasters)
