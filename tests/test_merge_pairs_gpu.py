"""The merge's pair search: folded rows, tiles and the cell grid find the same
contacts.

Merges of 33 spheres and more run on the block. Up to the pair tile (256
spheres with 32 threads, 1024 with more) the rows of the pair triangle are
folded in twos, above it they go tile by tile, and from the grid's minimum on
through hashed cells. Aggregates of odd and even sizes around 32, 64, 256 and
1024 merged spheres must end in the same bits and contact counts every way.
"""
import numpy as np
import pytest

from mcac_gb300 import Batch, PhysicalModel, synthetic_state
from mcac_gb300.api import set_merge_grid_min

CASES = {
    # spheres, aggregates, largest, steps
    "33 to 36": (680, 40, 17, 300),
    "63 to 66": (1280, 40, 32, 300),
    "254 to 258": (1536, 12, 128, 300),
    "500 to 515": (2056, 8, 257, 200),
    "1020 to 1030": (2056, 4, 514, 300),
}


def model(n, seed):
    return PhysicalModel(text=(
        f"[monomers]\nnumber = {n}\nmean_diameter = 30\ndispersion_diameter = 1.3\ninitialisation_mode = lognormal\n"
        f"[environment]\nvolume_fraction = 8e-3\ntemperature = 1700\n[limits]\nnumber_of_aggregates = 1\n"
        f"[numerics]\nrandom_seed = {seed}\nwith_domain_duplication = false\n"))


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [32, 128, 512])
@pytest.mark.parametrize("name", list(CASES))
def test_pair_searches_agree(name, threads):
    n, na, largest, steps = CASES[name]
    models = [model(n - k, 700 + k) for k in range(3)]
    states = [synthetic_state(m, na, max(largest, -(-int(m.params.n_monomeres) // na))) for m in models]
    runs = []
    for grid_min, nt in ((2, 128), (1 << 30, threads)):
        before = set_merge_grid_min(grid_min)
        try:
            with Batch(models, states=states) as b:
                b.threads = nt
                b.run(max_steps=steps, steps_per_launch=steps)
                st = b.stats()
                assert np.all(st["status"] == 0)
                runs.append((st, b.store_all(), b.work()))
        finally:
            set_merge_grid_min(before)
    (ref_st, ref, ref_work), (st, snaps, work) = runs
    assert st["events"].sum() > 0
    for f in ("steps", "events", "n_aggregates"):
        assert np.array_equal(st[f], ref_st[f]), f
    for s1, s2 in zip(snaps, ref):
        assert np.array_equal(s1.spheres.view(np.int64), s2.spheres.view(np.int64))
        assert np.array_equal(s1.aggregates.view(np.int64), s2.aggregates.view(np.int64))
        assert np.array_equal(s1.members, s2.members)
    for f in ("merged_spheres", "merge_pairs"):
        assert work[f] == ref_work[f], f
