"""A replay of a captured chain takes about as long as the eager call: it saves
the read-backs and pays for headroom.  What it must not lose is the overlap of
the two emission kernels.  Host times, the two in turn, the shortest of each."""
import time

import pytest

import oracle
from compare import compare
from ochre_gb300 import DeviceBatch, GpuContext, workloads

pytestmark = pytest.mark.gpu


def _times(batch, n=15):
    """(eager, replay) seconds, after both gave the oracle's output."""
    import torch
    exp = oracle.run(batch, threads=16)
    ctx = GpuContext(0, chain_only=True)
    try:
        db = DeviceBatch(batch)
        g = ctx.graph(db)
        runs = [lambda: ctx.rasterize_device(db), g.launch]
        for f in runs:
            compare(ctx.device_result_to_numpy(f(), batch.n_rasters), exp, batch.n_rasters)
        best = [1e9, 1e9]
        for _ in range(n):
            for k, f in enumerate(runs):
                torch.cuda.synchronize()
                t = time.perf_counter()
                f()
                torch.cuda.synchronize()
                best[k] = min(best[k], time.perf_counter() - t)
        g.close()
        return best
    finally:
        ctx.close()


def test_replay_overlaps_long_and_short_lines():
    """1,000 uneven paths: some 0.4 ms each for the few long lines and the many short
    ones, of 1.8 ms; one after the other a replay took 1.18 times the eager call."""
    eager, replay = _times(workloads.uneven_mix(n_paths=1000, seed=3))
    assert replay < 1.1 * eager, (eager, replay)
