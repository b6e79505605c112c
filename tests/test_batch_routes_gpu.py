"""Which kernels answer a batch of queries does not show in the answers.

Warps first with the rest by blocks, blocks of 256 threads, or blocks of 128:
chosen from the number of queries and the mean number of spheres per
aggregate. Batches on both sides of each line, with the same questions at
other places of the batch, against the queries asked one at a time.
"""
import numpy as np
import pytest

from mcac_gb300 import AggregatList, PhysicalModel, init_state, synthetic_state
from mcac_gb300.snapshot import A
from mcac_gb300.workloads import random_directions

FIELDS = ("moving_sphere", "other_sphere", "moving_aggregate", "other_aggregate")


@pytest.mark.gpu
@pytest.mark.parametrize("spheres, aggregates, largest", [(1500, 1500, 1), (1500, 300, 9), (1515, 300, 9),
                                                          (3000, 300, 30), (6000, 40, 400), (9000, 6, 3000)])
@pytest.mark.parametrize("n", [1, 2, 31, 639, 1216, 1217, 1999, 2000, 2001, 4000])
def test_batches_answer_like_single_queries(spheres, aggregates, largest, n):
    model = PhysicalModel(text=(
        f"[monomers]\nnumber = {spheres}\nmean_diameter = 30\ndispersion_diameter = 1.25\n"
        f"initialisation_mode = lognormal\n[environment]\nvolume_fraction = 5e-3\ntemperature = 1700\n"
        f"[numerics]\nrandom_seed = 77\nwith_domain_duplication = false\n"))
    state = init_state(model) if largest == 1 else synthetic_state(model, aggregates, largest)
    rng = np.random.Generator(np.random.PCG64(n))
    asked = min(n, 48)
    src = rng.integers(0, int(state.state.n_aggregates), asked)
    dirs = random_directions(rng, asked)
    far = np.where(np.arange(asked) % 2 == 0, state.aggregates[A["lpm"], src], 0.4 * state.state.box_length)
    at = rng.permutation(np.arange(n) % asked)  # question k stands wherever at == k
    with AggregatList(model, state) as box:
        out, _ = box.distance_to_next_contacts(src[at], dirs[at], far[at])
        one = [box.distance_to_next_contact(int(s), d, float(f)) for s, d, f in zip(src, dirs, far)]
    distance = np.array([o.distance for o in one])
    assert np.array_equal(out["distance"].view(np.int64), distance[at].view(np.int64))
    hit = np.isfinite(distance[at])
    assert n < 639 or hit.any()
    for f in FIELDS:
        assert np.array_equal(out[f][hit], np.array([getattr(o, f) for o in one])[at][hit]), f
