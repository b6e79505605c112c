"""Rounds that a limit cuts: few steps left in a launch, and the limit on the
steps without event.

A launch takes its first 64 steps one after another and at least sixteen
rounds after them, whatever their pace. So launches a few steps longer than
64 end with rounds of fewer steps than there are warps, and limits a little
above 64 on the steps without event are reached inside a round. Each case
checks that rounds of more than one step were committed, and that the run
ends in the bits of the steps one after another.
"""
import numpy as np
import pytest

from mcac_gb300 import Batch
from test_round_steps_gpu import assert_same, model

ALONE = 64


def run(models, threads, steps, chunk):
    with Batch(models) as b:
        b.threads = threads
        b.run(max_steps=steps, steps_per_launch=chunk)
        return (b.stats(), b.store_all(), b.work()), b.rounds()


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("more", [1, 2, 3, 6, 7, 8, 13, 15])
@pytest.mark.parametrize("ppm", [20, 5000])
def test_few_steps_left_in_a_launch(ppm, more, threads):
    models = [model(300 + k, 600 + k, ppm) for k in range(4)]
    launches = 12
    chunk = ALONE + more
    ref, none = run(models, 32, launches * chunk, chunk)
    assert none == (0, 0)
    got, (rounds, steps) = run(models, threads, launches * chunk, chunk)
    # (at 5000 ppm a query reads more cells than a warp's: most rounds leave
    # their first step to the block and commit nothing themselves)
    assert rounds > 0 and (steps > rounds or more == 1 or ppm == 5000)
    if more == 1:  # nothing but rounds of one step
        assert steps <= rounds
    assert_same(got, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("limit", [ALONE + k for k in (1, 2, 3, 5, 6, 7, 8, 9, 20)])
def test_a_limit_on_steps_without_event_inside_a_round(limit, threads):
    # 2 ppm: the first event comes hundreds of steps after the start
    models = [model(300 + k, 620 + k, 2, limits=f"n_iter_without_event = {limit}\n") for k in range(6)]
    ref, _ = run(models, 32, 4000, 4000)
    assert np.all(ref[0]["finished"] != 0) and (ref[0]["steps"] == limit).any()
    got, (rounds, steps) = run(models, threads, 4000, 4000)
    assert rounds > 0 and (steps > rounds or limit == ALONE + 1)
    assert_same(got, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [256, 512])
def test_rounds_with_events_commit_several_steps(threads):
    models = [model(400 + k, 640 + k, 2000) for k in range(4)]
    ref, _ = run(models, 32, 3000, 1000)
    got, (rounds, steps) = run(models, threads, 3000, 1000)
    assert ref[0]["events"].sum() > 100 and steps > 1.2 * rounds > 0
    assert_same(got, ref)
