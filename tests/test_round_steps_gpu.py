"""Steps taken in rounds (blocks of 256 threads and more) against one warp.

A round answers the next steps of a box at once and commits them in order up
to the first that another could have changed; a box on 32 threads takes its
steps one after another. Both must end in the same bits wherever a run can
stop: launches of any length (also shorter than a round), a limit on the
steps without event, a limit on the physical time that falls inside a round,
boxes whose sweeps always meet (dense, few aggregates), boxes whose steps
leave their cells together, and boxes that run to their end.
"""
import numpy as np
import pytest

from mcac_gb300 import Batch, PhysicalModel


def model(n, seed, ppm, n_div=10, limits=""):
    return PhysicalModel(text=(
        f"[monomers]\nnumber = {n}\nmean_diameter = 30\ndispersion_diameter = 1.3\ninitialisation_mode = lognormal\n"
        f"[environment]\nvolume_fraction = {ppm * 1e-6!r}\ntemperature = 1700\n"
        f"[limits]\nnumber_of_aggregates = 1\n{limits}"
        f"[numerics]\nn_verlet_divisions = {n_div}\nrandom_seed = {seed}\nwith_domain_duplication = false\n"))


CASES = {
    # spheres, ppm, Verlet cells per axis, limits, steps, steps per launch
    "sparse": (500, 10, 10, "", 1501, 500),
    "launches shorter than a round": (300, 500, 10, "", 199, 3),
    "dense": (300, 30000, 6, "", 600, 601),
    "two spheres": (2, 2000, 4, "", 400, 37),
    "one cell an axis": (60, 2000, 1, "", 700, 350),
    "many cells": (400, 300, 40, "", 900, 300),
    "to the end": (40, 20000, 8, "", 6000, 2000),
    "steps without event": (200, 300, 10, "n_iter_without_event = 23\n", 4000, 1000),
    "one step without event": (200, 300, 10, "n_iter_without_event = 1\n", 50, 50),
}


def run(models, threads, steps, chunk):
    with Batch(models) as b:
        b.threads = threads
        b.run(max_steps=steps, steps_per_launch=chunk)
        st = b.stats()
        return st, b.store_all(), b.work()


def assert_same(one, other):
    (st, snaps, work), (ref_st, ref, ref_work) = one, other
    for f in ("status", "steps", "events", "n_aggregates", "finished"):
        assert np.array_equal(st[f], ref_st[f]), f
    assert np.array_equal(st["time"].view(np.int64), ref_st["time"].view(np.int64))
    for s1, s2 in zip(snaps, ref):
        assert s1.maxradius == s2.maxradius
        assert np.array_equal(s1.spheres.view(np.int64), s2.spheres.view(np.int64))
        assert np.array_equal(s1.aggregates.view(np.int64), s2.aggregates.view(np.int64))
        assert np.array_equal(s1.members, s2.members) and np.array_equal(s1.sphere_label, s2.sphere_label)
    for f in ("queries", "merges", "translates", "mov_spheres", "candidates", "cand_spheres", "refined",
              "merged_spheres", "merge_pairs"):
        assert work[f] == ref_work[f], f


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("name", list(CASES))
def test_rounds_equal_steps_one_after_another(name, threads):
    n, ppm, n_div, limits, steps, chunk = CASES[name]
    models = [model(n + (k if n > 2 else 0), 500 + k, ppm, n_div, limits) for k in range(4)]
    ref = run(models, 32, steps, chunk)
    assert np.all(ref[0]["status"] == 0) and ref[0]["steps"].sum() > 0
    assert_same(run(models, threads, steps, chunk), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("at", [130, 131, 132, 133, 134, 135, 136, 300])
def test_a_time_limit_inside_a_round(threads, at):
    plain = [model(400, 540 + k, 50) for k in range(3)]
    reached = run(plain, 32, at, at)[0]["time"]
    models = [model(400, 540 + k, 50, limits=f"physical_time = {float(t)!r}\n") for k, t in enumerate(reached)]
    ref = run(models, 32, 2 * at, 2 * at)
    assert np.all(ref[0]["finished"] != 0)
    assert_same(run(models, threads, 2 * at, 2 * at), ref)
