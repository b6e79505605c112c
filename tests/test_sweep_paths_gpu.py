"""Contact queries at the lengths where the swept test changes its route.

A sweep shorter than the box takes the short form of the swept test (one
periodic image, comparisons of bit patterns); one whose zone reaches the box
length takes the general one (several images), and Verlet ranges whose ends
lie near a cell boundary are decided in FP64. Every answer must have the
oracle's bits: same distance, spheres and aggregate. The lengths are given in
box lengths around the switch; axis-aligned directions from a centre put the
range's ends on and next to cell boundaries.
"""
import numpy as np
import pytest

from conftest import load_golden
from mcac_gb300 import AggregatList, PhysicalModel
from mcac_gb300.snapshot import A, Snapshot
from mcac_gb300.workloads import random_directions
from oracle import oracle_py as O


def check(box, ob, label, direction, distance):
    got = box.distance_to_next_contact(int(label), direction, float(distance))
    ref = ob.distance_to_next_contact(int(label), direction, float(distance))
    assert np.float64(got.distance).view(np.int64) == np.float64(ref.distance).view(np.int64)
    if np.isfinite(ref.distance):
        assert (got.moving_sphere, got.other_sphere, got.other_aggregate) == (
            ref.moving_sphere, ref.other_sphere, ref.other_aggregate)
    return np.isfinite(ref.distance)


@pytest.mark.gpu
@pytest.mark.parametrize("fixture", ["c1_q5000.npz", "ln_late.npz"])
@pytest.mark.parametrize("boxes", [0.0, 1e-3, 0.1, 0.45, 0.499, 0.55, 0.9, 0.999, 1.001, 2.5])
def test_sweeps_around_the_box_length_match_the_oracle(fixture, boxes):
    g = load_golden(fixture)
    snap = Snapshot.from_npz(g, "s_")
    ini = str(g["ini"])
    ob = O.OracleBox(ini, snap)
    rng = np.random.Generator(np.random.PCG64(int(1000 * boxes) + 7))
    hits = 0
    with AggregatList(PhysicalModel(text=ini), snap) as box:
        for label, d in zip(rng.integers(0, snap.na, 12), random_directions(rng, 12)):
            hits += check(box, ob, label, d, boxes * snap.box_length)
    assert hits > 0 or boxes < 0.9


@pytest.mark.gpu
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("off", [0.0, 1e-15, -1e-15, 1e-7, -1e-7, 1e-5])
def test_verlet_ranges_ending_on_cell_boundaries_match_the_oracle(axis, off):
    g = load_golden("c1_q5000.npz")
    snap = Snapshot.from_npz(g, "s_")
    ini = str(g["ini"])
    ob = O.OracleBox(ini, snap)
    cell = snap.box_length / snap.n_div
    with AggregatList(PhysicalModel(text=ini), snap) as box:
        for label in range(0, snap.na, max(1, snap.na // 12)):
            for sign in (1.0, -1.0):
                d = np.zeros(3)
                d[axis] = sign
                # the length that takes the range's leading end to a boundary
                x, reach = snap.aggregates[A["x"] + axis, label], snap.aggregates[A["rmax"], label] + snap.maxradius
                end = x + sign * reach
                edge = (np.floor(end / cell) + (2 if sign > 0 else -1)) * cell
                check(box, ob, label, d, abs(edge - end) + off * cell)
