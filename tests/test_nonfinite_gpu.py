"""Contact queries on boxes that hold infinite and NaN coordinates.

The swept test compares bit patterns, and a NaN made by the GPU has its sign
bit set (an infinite coordinate makes one in the periodic distance), so it
must not order below the contact distance: a sphere without a finite place
touches nothing, as in the oracle. The FP32 screens drop such spheres for
short sweeps; a sweep of more than a box length hands every pair to the swept
test. Single queries and both forms of a batch.
"""
import numpy as np
import pytest

from conftest import load_golden
from mcac_gb300 import AggregatList, Batch, PhysicalModel, StateBuffers
from mcac_gb300._lib import MCACError
from mcac_gb300.snapshot import A, S, Snapshot
from mcac_gb300.workloads import random_directions
from oracle import oracle_py as O

NEGATIVE_NAN = np.array([-0x8000000000000], dtype=np.int64).view(np.float64)[0]


@pytest.mark.gpu
@pytest.mark.parametrize("centres", [False, True])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, NEGATIVE_NAN], ids=["inf", "-inf", "nan", "-nan"])
@pytest.mark.parametrize("boxes", [0.1, 1.2])
@pytest.mark.parametrize("fixture", ["c1_q5000.npz", "ln_late.npz"])
def test_spheres_without_a_place_touch_nothing(fixture, boxes, value, centres):
    g = load_golden(fixture)
    snap = Snapshot.from_npz(g, "s_")
    ini = str(g["ini"])
    rng = np.random.Generator(np.random.PCG64(int(10 * boxes) + 31))
    lost = np.arange(1, snap.na, 3)  # these aggregates' spheres lose a coordinate
    # (the oracle's wrap loops end for a NaN only, and its cells need finite
    # centres: it keeps those, and has a NaN for every lost coordinate)
    ref_snap = snap.copy()
    for a in lost:
        snap.spheres[S["x"] + a % 3, snap.members_of(a)] = value
        ref_snap.spheres[S["x"] + a % 3, snap.members_of(a)] = np.nan
    ob = O.OracleBox(ini, ref_snap)
    if centres:
        snap.aggregates[A["x"] + lost % 3, lost] = value
    labels = rng.choice(np.setdiff1d(np.arange(snap.na), lost), 12)
    dirs = random_directions(rng, 12)
    length = boxes * snap.box_length
    ref = [ob.distance_to_next_contact(int(l), d, length) for l, d in zip(labels, dirs)]
    with AggregatList(PhysicalModel(text=ini), snap) as box:
        one = [box.distance_to_next_contact(int(l), d, length) for l, d in zip(labels, dirs)]
        few, _ = box.distance_to_next_contacts(labels, dirs, np.full(12, length))
        many, _ = box.distance_to_next_contacts(np.tile(labels, 60), np.tile(dirs, (60, 1)), np.full(720, length))
    for k, r in enumerate(ref):
        got = [one[k]] + [_Row(b[k]) for b in (few, many[:12], many[-12:])]
        for c in got:
            assert np.float64(c.distance).view(np.int64) == np.float64(r.distance).view(np.int64)
            if np.isfinite(r.distance):
                assert (c.moving_sphere, c.other_sphere, c.other_aggregate) == (
                    r.moving_sphere, r.other_sphere, r.other_aggregate)
    assert any(np.isfinite(r.distance) for r in ref) or boxes < 1.0


class _Row:
    def __init__(self, row):
        for f in ("distance", "moving_sphere", "other_sphere", "other_aggregate"):
            setattr(self, f, row[f])


@pytest.mark.gpu
@pytest.mark.parametrize("boxes", [0, 1, -1, 7, -40, 100000])
@pytest.mark.parametrize("fixture", ["c1_q5000.npz", "ln_late.npz"])
def test_one_query_and_a_batch_agree_on_centres_outside_the_box(fixture, boxes):
    """A state's centres are not checked when it is loaded. The source of the
    query and its spheres lie whole boxes away: its cells are taken modulo the
    grid, and both forms of the query find the same (the Verlet grid files the
    centre under its nearest cell, so most often: that it is not listed)."""
    g = load_golden(fixture)
    snap = Snapshot.from_npz(g, "s_")
    rng = np.random.Generator(np.random.PCG64(77))
    labels = rng.choice(snap.na, 10, replace=False)
    for l in labels:
        snap.aggregates[A["x"]:A["z"] + 1, l] += boxes * snap.box_length
        snap.spheres[:3, snap.members_of(l)] += boxes * snap.box_length
    found = 0
    with AggregatList(PhysicalModel(text=str(g["ini"])), snap) as box:
        for l, d in zip(labels, random_directions(rng, 10)):
            for length in (1e-3 * snap.box_length, 0.3 * snap.box_length, snap.box_length):
                got = []
                for ask in (lambda: box.distance_to_next_contact(int(l), d, length),
                            lambda: _Row(box.distance_to_next_contacts([l], [d], [length])[0][0])):
                    try:
                        c = ask()
                        got.append((c.distance, c.moving_sphere, c.other_sphere, c.other_aggregate))
                    except MCACError as e:
                        got.append(e.code)
                assert got[0] == got[1]
                found += not isinstance(got[0], int)
    assert boxes != 0 or found == 30


@pytest.mark.gpu
@pytest.mark.parametrize("collisions", ["true", "false"])
@pytest.mark.parametrize("value", [np.inf, np.nan, NEGATIVE_NAN], ids=["inf", "nan", "-nan"])
def test_steps_without_a_finite_length_meet_nothing(value, collisions):
    models = [PhysicalModel(text=(
        f"[monomers]\nnumber = {n}\nmean_diameter = 30\ndispersion_diameter = 1.3\ninitialisation_mode = lognormal\n"
        f"[environment]\nvolume_fraction = 5e-3\ntemperature = 1700\n[limits]\nnumber_of_aggregates = 1\n"
        f"[numerics]\nrandom_seed = {n}\nwith_domain_duplication = false\nwith_collisions = {collisions}\n"))
        for n in (60, 90)]
    with Batch(models) as b:
        snaps = b.store_all()
    for s in snaps:
        s.aggregates[A["lpm"], ::3] = value
    ends = []
    for threads in (32, 128, 256, 512):
        with Batch(models, states=[StateBuffers.from_snapshot(s) for s in snaps]) as b:
            b.threads = threads
            b.run(max_steps=100, steps_per_launch=100)
            st = b.stats()
            assert np.all(st["status"] == 0) and np.all(st["steps"] == 100)
            assert np.array_equal(st["events"], [s.na for s in snaps] - st["n_aggregates"])
            ends.append((st, b.store_all()))
    for st, out in ends[1:]:
        for f in ("events", "n_aggregates", "time"):
            assert np.array_equal(st[f], ends[0][0][f]), f
        for x, y in zip(out, ends[0][1]):
            assert np.array_equal(x.spheres, y.spheres, equal_nan=True)
            assert np.array_equal(x.members, y.members) and np.array_equal(x.sphere_label, y.sphere_label)
    assert collisions == "true" or not ends[0][0]["events"].any()
