"""Splits of oxidising aggregates give the same parts in every run.

An aggregate's connected parts come from a disjoint-set forest that all
threads build and walk at once. Aggregates joined from several grown ones, in
a shuffled member order (deep forests), fall apart in the first step: each
part must be one of the networks that were joined, the part of the first
member keeps the aggregate's place, and all copies of the box must end in the
same bits, whatever the order in which their threads ran.
"""
import numpy as np
import pytest

from mcac_gb300 import Batch, synthetic_state
from mcac_gb300.snapshot import A, S
from test_update_paths_gpu import model


def joined(snap, groups, seed):
    """The snapshot with its aggregates joined into 'groups' ones, each holding
    several separate networks, members in a shuffled order."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = snap.copy()
    off = snap.member_offsets()
    members, counts, cols = [], [], []
    for g in range(groups):
        own = [snap.members[off[a]:off[a + 1]] for a in range(g, snap.na, groups)]
        m = rng.permutation(np.concatenate(own))
        p = snap.spheres[:3, m]
        for l in range(3):
            out.spheres[S["rx"] + l, m] = p[l] - p[l, 0]
        centre = p.mean(axis=1)
        col = snap.aggregates[:, g].copy()
        col[[A["x"], A["y"], A["z"]]] = np.mod(centre, snap.box_length)
        col[A["rmax"]] = (np.sqrt(((p - centre[:, None]) ** 2).sum(0)) + snap.spheres[S["r"], m]).max()
        out.sphere_label[m] = g
        members.append(m)
        counts.append(len(m))
        cols.append(col)
    out.members, out.n_spheres = np.concatenate(members), np.array(counts, dtype=np.int64)
    out.aggregates = np.ascontiguousarray(np.stack(cols, axis=1))
    out.maxradius = max(snap.maxradius, out.aggregates[A["rmax"]].max())
    return out


def networks(snap, m):
    """The connected networks of touching spheres among the spheres m."""
    p, r = snap.spheres[:3, m], snap.spheres[S["r"], m]
    d = p[:, :, None] - p[:, None, :]
    d -= snap.box_length * np.round(d / snap.box_length)
    touch = (d ** 2).sum(0) - (r[:, None] + r[None, :]) ** 2 <= 1e-28
    left, out = set(range(len(m))), []
    while left:
        todo = [left.pop()]
        seen = set(todo)
        while todo:
            new = left.intersection(np.flatnonzero(touch[todo.pop()]).tolist())
            left -= new
            seen |= new
            todo += new
        out.append(frozenset(int(m[k]) for k in seen))
    return set(out)


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [32, 128, 512])
def test_every_copy_splits_into_the_joined_networks(threads):
    grow = model(900, 17, 4.0, limit=0)
    burn = model(900, 17, -1e-9, limit=0, extra="with_collisions = false\n")
    with Batch([grow], states=[synthetic_state(grow, 12, 200)]) as b:
        b.run(max_steps=30, steps_per_launch=30)
        start = joined(b.store(0), 3, 5)
    copies = 200
    with Batch([burn] * copies, states=[start] * copies) as b:
        b.threads = threads
        b.run(max_steps=1, steps_per_launch=1)
        assert np.all(b.stats()["status"] == 0)
        ends = b.store_all()
    first = ends[0]
    parts = [first.members[o:o + n] for o, n in zip(first.member_offsets(), first.n_spheres)]
    assert first.na > start.na
    lists = [start.members[o:o + n] for o, n in zip(start.member_offsets(), start.n_spheres)]
    assert {frozenset(p.tolist()) for p in parts} == set().union(*(networks(first, m) for m in lists))
    place = np.empty(start.ns, dtype=np.int64)  # of each sphere in the joined lists
    place[start.members] = np.arange(start.ns)
    assert all(np.all(np.diff(place[p]) > 0) for p in parts)  # list order kept
    assert all(first.sphere_label[m[0]] == g for g, m in enumerate(lists))
    for s in ends[1:]:
        assert np.array_equal(s.sphere_label, first.sphere_label) and np.array_equal(s.members, first.members)
        assert np.array_equal(s.spheres.view(np.int64), first.spheres.view(np.int64))
        assert np.array_equal(s.aggregates.view(np.int64), first.aggregates.view(np.int64))
