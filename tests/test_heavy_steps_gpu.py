"""Boxes whose queries are mostly the block's.

Dense boxes of few aggregates: a warp counts a query's pairs before its FP64
filter and leaves it early, and after some such queries in a row the next ones
go to the block without a try, all but every eighth. Runs must have the
bits of the block's own steps, with sources on both sides of the size from
which this holds (8 spheres) and the small and the large mixed.
"""
import numpy as np
import pytest

from mcac_gb300 import Batch, synthetic_state
from test_round_steps_gpu import assert_same, model


def run(models, states, threads, blocks, steps, chunk):
    with Batch(models, states=states) as b:
        b.threads = threads
        b.speculation = blocks
        b.run(max_steps=steps, steps_per_launch=chunk)
        return b.stats(), b.store_all(), b.work()


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [32, 128, 256, 512])
@pytest.mark.parametrize("spheres, aggregates, largest, ppm", [(200, 8, 80, 8000), (300, 20, 60, 8000),
                                                               (150, 20, 8, 12000), (170, 20, 9, 12000),
                                                               (600, 60, 200, 10000), (900, 300, 40, 8000)])
@pytest.mark.parametrize("chunk", [250, 90])
def test_runs_have_the_blocks_bits(spheres, aggregates, largest, ppm, threads, chunk):
    models = [model(spheres + 3 * k, 800 + k, ppm) for k in range(4)]
    states = [synthetic_state(m, aggregates, largest) for m in models]
    ref = run(models, states, 128, 2, 250, chunk)
    assert np.all(ref[0]["status"] == 0) and ref[0]["events"].sum() > 0
    assert_same(run(models, states, threads, 1, 250, chunk), ref)
