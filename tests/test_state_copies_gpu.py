"""States of many boxes in page-locked arrays are copied by one kernel.

From two boxes on, where every array lies in page-locked blocks of the library,
loading and storing go through k_copy_pieces: chunks of 32 KiB, 16 bytes at a
time where both ends are 16-byte aligned, else 8. What it moves must be what
the driver's copies move for the same boxes in ordinary arrays: arrays below,
at and above a multiple of the chunk, boxes of one and two spheres, odd
offsets in a shared block, a box with an array elsewhere, fewer aggregates at
the end than at the start, room for more than is stored, and an empty box.
"""
import numpy as np
import pytest

from mcac_gb300 import Batch, PhysicalModel, StateBuffers
from mcac_gb300._lib import State, _PinnedBlock, f64, i64, ptr

FIELDS = ("spheres", "sphere_label", "aggregates", "n_spheres", "members")


def model(n, seed, extra=""):
    return PhysicalModel(text=(
        f"[monomers]\nnumber = {n}\nmean_diameter = 30\ndispersion_diameter = 1.3\ninitialisation_mode = lognormal\n"
        f"[environment]\nvolume_fraction = 3e-3\ntemperature = 1700\n{extra}"
        f"[limits]\nnumber_of_aggregates = 1\n[numerics]\nrandom_seed = {seed}\nwith_domain_duplication = false\n"))


def states_of(models, steps=0):
    with Batch(models) as b:
        if steps:
            b.run(max_steps=steps, steps_per_launch=steps)
        return b.store_all(raw=True)


def page_locked(src, gap=0, room=0):
    """Copies of the states in one page-locked block, 'gap' words of 8 bytes
    between arrays and room for 'room' more spheres and aggregates."""
    sizes = [(int(s.state.n_spheres), int(s.state.n_aggregates)) for s in src]
    words = sum(11 * (ns + room) + 22 * (na + room) + 5 * gap + gap for ns, na in sizes) + 8
    buf = _PinnedBlock(8 * words).buffer()
    at, out = gap, []
    for s, (ns, na) in zip(src, sizes):
        b = StateBuffers(1, 1)
        for name, dt, shape in StateBuffers._layout(ns + room, na + room):
            count = int(np.prod(shape))
            a = np.frombuffer(buf, dtype=dt, count=count, offset=8 * at).reshape(shape)
            at += count + gap
            a[...] = -7
            if room == 0:
                a[...] = np.asarray(getattr(s, name)).reshape(-1)[:count].reshape(shape)
            setattr(b, name, a)
        b.state = State(ns + room, na + room, s.state.n_verlet_divisions, s.state.box_length, s.state.maxradius,
                        s.state.time, ptr(b.spheres, f64), ptr(b.sphere_label, i64), ptr(b.aggregates, f64),
                        ptr(b.n_spheres, i64), ptr(b.members, i64))
        out.append(b)
    return out


def assert_equal(one, other):
    assert len(one) == len(other)
    for x, y in zip(one, other):
        ns, na = int(x.state.n_spheres), int(x.state.n_aggregates)
        assert (ns, na) == (int(y.state.n_spheres), int(y.state.n_aggregates))
        assert (x.state.box_length, x.state.maxradius, x.state.time) == (
            y.state.box_length, y.state.maxradius, y.state.time)
        for f, count in zip(FIELDS, (9 * ns, ns, 21 * na, na, ns)):
            a, b = (np.asarray(getattr(s, f)).reshape(-1)[:count].view(np.int64) for s in (x, y))
            assert np.array_equal(a, b), f


# spheres of a box: 72 B and 8 B each, aggregates 168 B: around 32 KiB chunks
SIZES = [1, 2, 3, 195, 196, 455, 456, 911, 4095, 4096, 4097, 1365, 586, 64, 65, 8191, 17, 18, 390, 1000]


@pytest.mark.gpu
@pytest.mark.parametrize("boxes", [1, 2, 3, 17, 20])
@pytest.mark.parametrize("gap", [0, 1, 3])
@pytest.mark.parametrize("steps", [0, 60])
def test_page_locked_states_are_those_of_ordinary_arrays(boxes, gap, steps):
    models = [model(n, 40 + k) for k, n in enumerate(SIZES[:boxes])]
    plain = states_of(models, steps)
    locked = page_locked(plain, gap=gap)
    ends = []
    for states in (plain, locked):
        with Batch(models, states=states) as b:
            held = b.store_all(raw=True), b.store_all(raw=True, out=page_locked(plain, gap=gap, room=5))
            assert_equal(held[0], plain)
            assert_equal(held[1], plain)
            b.run(max_steps=80, steps_per_launch=80)
            # fewer aggregates now: into new arrays, page-locked and not, and
            # into arrays of the sizes at the start
            ends += [b.store_all(raw=True), b.store_all(raw=True, pinned=True),
                     b.store_all(raw=True, out=page_locked(plain, gap=gap))]
    for e in ends[1:]:
        assert_equal(e, ends[0])
    if boxes >= 17:
        assert sum(int(s.state.n_aggregates) for s in ends[0]) < sum(int(s.state.n_aggregates) for s in plain)


@pytest.mark.gpu
@pytest.mark.parametrize("which", FIELDS)
def test_one_array_elsewhere_takes_the_other_way(which):
    models = [model(n, 70 + k) for k, n in enumerate(SIZES[:18])]
    plain = states_of(models, 30)
    locked = page_locked(plain)
    # the ninth box has one array in ordinary memory
    setattr(locked[8], which, np.array(getattr(locked[8], which)))
    setattr(locked[8].state, {"n_spheres": "n_spheres_per_aggregate"}.get(which, which),
            ptr(getattr(locked[8], which), f64 if which in ("spheres", "aggregates") else i64))
    with Batch(models, states=locked) as b:
        assert_equal(b.store_all(raw=True), plain)
        assert_equal(b.store_all(raw=True, out=locked), plain)


@pytest.mark.gpu
def test_boxes_left_empty_store_nothing():
    # monodisperse monomers reach rp_min together: every other box ends empty
    burn = ("[surface_growth]\nwith_surface_reactions = true\nflux_surfgrowth = -0.5\n[oxidation]\nrp_min = 1e-8\n")
    models = [PhysicalModel(text=(
        f"[monomers]\nnumber = {30 + k}\nmean_diameter = 30\ndispersion_diameter = 1.0\n"
        f"initialisation_mode = lognormal\n[environment]\nvolume_fraction = 1e-3\ntemperature = 1700\n"
        f"{burn if k % 2 else ''}[limits]\nnumber_of_aggregates = {0 if k % 2 else 25}\n"
        f"[numerics]\nrandom_seed = {90 + k}\nwith_domain_duplication = false\n")) for k in range(18)]
    with Batch(models) as b:
        room = page_locked(b.store_all(raw=True))
        b.run(max_steps=0, steps_per_launch=20000)
        st = b.stats()
        plain = b.store_all(raw=True)
        locked = b.store_all(raw=True, out=room)
    assert np.all(st["status"] == 0) and np.all(st["n_aggregates"][1::2] == 0) and np.all(st["n_aggregates"][::2] > 0)
    assert_equal(locked, plain)
    assert all(int(s.state.n_spheres) == 0 for s in locked[1::2])
