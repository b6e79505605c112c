"""The work counters do not depend on how the loop took its steps.

With 256 threads and more the form of the loop is chosen by the pace of both
forms as they run, and a round's queries read the neighbour lists as they
stand at its start. The counts of aggregates scanned and cells visited (the
benchmark's model of bytes) must be those of the steps one after another all
the same: on the fine grid, on the Verlet cells, and on the live list.
"""
import pytest

from test_round_steps_gpu import CASES, model, run

MORE = {
    # the Verlet cells are the finer grid, and most steps leave their cell
    "many Verlet cells": (300, 100, 60, "", 900, 450),
    "few aggregates": (140, 1000, 10, "", 3000, 1000),
}


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("name", ["sparse", "dense", "one cell an axis", "many cells", "to the end", *MORE])
def test_scanned_and_cells_equal_steps_one_after_another(name, threads):
    n, ppm, n_div, limits, steps, chunk = {**CASES, **MORE}[name]
    models = [model(n + k, 700 + k, ppm, n_div, limits) for k in range(6)]
    ref = run(models, 128, steps, chunk)[2]  # one after another, with the same live list
    assert ref["scanned"] > 0
    for _ in range(2):
        work = run(models, threads, steps, chunk)[2]
        for f in ("queries", "scanned", "cells", "candidates", "refined"):
            assert work[f] == ref[f], f
