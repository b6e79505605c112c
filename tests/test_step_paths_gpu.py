"""The device loop's one-warp steps against the block's routines.

Small steps run on one warp, larger ones (neighbour lists, candidates, sphere
pairs, moved or merged spheres above the one-warp limits) on the block;
speculative rounds (two blocks per box) run every step on the block's
routines. Both must end in the same bits with the same counts. The states
are synthetic aggregates whose sizes straddle the limits: 32 merged spheres,
64 moved ones, 1024 sphere pairs, 128 cells and 256 listed aggregates, and
boxes of one and two aggregates.
"""
import numpy as np
import pytest

from mcac_gb300 import Batch, PhysicalModel, synthetic_state
from mcac_gb300.api import set_live_list_max

COUNTS = ("queries", "merges", "translates", "mov_spheres", "candidates", "cand_spheres", "refined",
          "merged_spheres", "merge_pairs")


def model(n, seed, ppm, n_div=10, volsurf="none"):
    return PhysicalModel(text=(
        f"[monomers]\nnumber = {n}\nmean_diameter = 30\ndispersion_diameter = 1.3\ninitialisation_mode = lognormal\n"
        f"[environment]\nvolume_fraction = {ppm * 1e-6!r}\ntemperature = 1700\n"
        f"[surface_growth]\nvolsurf_method = {volsurf}\n"
        f"[limits]\nnumber_of_aggregates = 1\n[numerics]\nn_verlet_divisions = {n_div}\nrandom_seed = {seed}\n"
        f"with_domain_duplication = false\n"))


CASES = {
    # spheres, aggregates, largest, ppm, Verlet cells per axis, steps
    "pairs": (40, 20, 2, 8000, 10, 600),
    "merges of 30 to 34": (640, 40, 17, 8000, 10, 400),
    "moves of 60 to 68": (1300, 20, 68, 5000, 10, 300),
    "more than 1024 pairs": (1500, 10, 400, 5000, 10, 200),
    "crowded cells": (3000, 3000, 1, 20000, 3, 300),
    "crowded, small aggregates": (4000, 1300, 8, 20000, 4, 300),
    "many cells": (1200, 300, 30, 300, 40, 300),
    "two left": (60, 2, 40, 5000, 10, 400),
}


@pytest.mark.gpu
@pytest.mark.parametrize("live", [0, 128])
@pytest.mark.parametrize("threads", [32, 128, 512])
@pytest.mark.parametrize("name", list(CASES))
def test_one_warp_steps_equal_the_blocks(name, threads, live):
    n, na, largest, ppm, n_div, steps = CASES[name]
    models = [model(n + 7 * k, 300 + k, ppm, n_div) for k in range(3)]
    states = [synthetic_state(m, na, max(largest, -(-int(m.params.n_monomeres) // na))) for m in models]
    runs = []
    for blocks in (1, 2):
        before = set_live_list_max(live)
        try:
            with Batch(models, states=states) as b:
                b.threads = threads
                b.speculation = blocks
                b.run(max_steps=steps, steps_per_launch=steps // 3 + 1)
                st = b.stats()
                assert np.all(st["status"] == 0)
                runs.append((st, b.store_all(), b.work()))
        finally:
            set_live_list_max(before)
    (st, snaps, work), (ref_st, ref, ref_work) = runs
    for f in ("steps", "events", "n_aggregates", "finished"):
        assert np.array_equal(st[f], ref_st[f]), f
    assert np.array_equal(st["time"].view(np.int64), ref_st["time"].view(np.int64))
    assert st["events"].sum() > 0
    for s1, s2 in zip(snaps, ref):
        assert s1.maxradius == s2.maxradius
        assert np.array_equal(s1.spheres.view(np.int64), s2.spheres.view(np.int64))
        assert np.array_equal(s1.aggregates.view(np.int64), s2.aggregates.view(np.int64))
        assert np.array_equal(s1.members, s2.members) and np.array_equal(s1.sphere_label, s2.sphere_label)
    # (a round's queries see the state at its start, so the neighbours scanned,
    # though not the candidates, may differ)
    for f in COUNTS:
        assert work[f] == ref_work[f], f


@pytest.mark.gpu
@pytest.mark.parametrize("volsurf", ["caps", "alphas"])
def test_corrected_volumes_merge_on_the_block(volsurf):
    models = [model(300, 320 + k, 5000, volsurf=volsurf) for k in range(2)]
    runs = []
    for blocks in (1, 2):
        with Batch(models) as b:
            b.threads = 128
            b.speculation = blocks
            b.run(max_steps=800, steps_per_launch=800)
            runs.append((b.stats(), b.store_all()))
    assert np.array_equal(runs[0][0]["events"], runs[1][0]["events"]) and runs[0][0]["events"].sum() > 0
    for s1, s2 in zip(runs[0][1], runs[1][1]):
        assert np.array_equal(s1.aggregates.view(np.int64), s2.aggregates.view(np.int64))
