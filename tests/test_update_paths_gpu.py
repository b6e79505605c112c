"""The per-step update and the contact check of boxes with surface reactions.

A single sphere at its aggregate's centre takes a short form, aggregates of
up to 4 spheres are updated by a thread each and larger ones by a warp each,
32 spheres at a time; every field must have the bits of the reference's
sequential sums (restated in numpy: cumulative sums in list order, one
rounding per operation). Aggregate sizes straddle the limits. Oxidation's
contact networks are checked row by row over all warps, in shared memory up
to 2048 rows: every aggregate left must be one network, whatever the box and
the block size.
"""
import numpy as np
import pytest

from mcac_gb300 import Batch, PhysicalModel, synthetic_state
from mcac_gb300.snapshot import A, S


def model(n, seed, flux, limit=1, extra=""):
    return PhysicalModel(text=(
        f"[monomers]\nnumber = {n}\nmean_diameter = 30\ndispersion_diameter = 1.3\ninitialisation_mode = lognormal\n"
        f"[environment]\nvolume_fraction = 3e-3\ntemperature = 1700\n"
        f"[surface_growth]\nwith_surface_reactions = true\nflux_surfgrowth = {flux!r}\n"
        f"full_aggregate_update_frequency = 1\n[oxidation]\nrp_min = 2e-9\n"
        f"[limits]\nnumber_of_aggregates = {limit}\n[numerics]\nrandom_seed = {seed}\n"
        f"with_domain_duplication = false\n{extra}"))


def seq(x):
    return np.cumsum(x)[-1]


def wrap(p, L):
    while p < 0:
        p += L
    while p >= L:
        p -= L
    return p


def expected(snap, a):
    off = snap.member_offsets()
    m = snap.members[off[a]:off[a + 1]]
    r, v, s = (snap.spheres[S[f], m] for f in ("r", "volume", "surface"))
    rel = snap.spheres[[S["rx"], S["ry"], S["rz"]]][:, m]
    V = seq(v)
    c = [seq(rel[l] * v) / V for l in range(3)]
    d = [rel[l] - c[l] for l in range(3)]
    dc = np.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    brg = seq(v * (r * r))
    out = {"volume": V, "surface": seq(s), "rx": c[0], "ry": c[1], "rz": c[2], "rmax": np.max(r + dc),
           "rg": np.sqrt(abs((seq(v * (dc * dc)) + (3.0 / 5.0) * brg) / V)), "dp": 2 * seq(r) / float(len(m))}
    out["dg_over_dp"] = out["rg"] / (0.5 * out["dp"])
    for l, f in enumerate("xyz"):
        out[f] = wrap(snap.spheres[S[f], m[0]] + c[l], snap.box_length)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [32, 128, 512])
@pytest.mark.parametrize("spheres, aggregates, largest", [(90, 90, 1), (200, 60, 5), (330, 10, 33), (650, 10, 66),
                                                          (1200, 5, 300)])
def test_updated_fields_have_the_bits_of_the_sequential_sums(spheres, aggregates, largest, threads):
    m = model(spheres, 11, 1e-2)
    states = None if largest == 1 else [synthetic_state(m, aggregates, largest)]
    with Batch([m], states=states) as b:
        b.threads = threads
        b.run(max_steps=25, steps_per_launch=25)
        assert np.all(b.stats()["status"] == 0)
        snap = b.store(0)
    for a in range(snap.na):
        for f, v in expected(snap, a).items():
            assert np.float64(v).view(np.int64) == snap.aggregates[A[f], a].view(np.int64), (a, snap.n_spheres[a], f)


@pytest.mark.gpu
@pytest.mark.parametrize("spheres, aggregates, largest, steps", [(60, 20, 6, 40), (700, 6, 300, 40), (3000, 20, 400, 5)])
def test_oxidised_aggregates_stay_one_network_each(spheres, aggregates, largest, steps):
    grow, burn = model(spheres, 13, 4.0, limit=0), model(spheres, 13, -20.0, limit=0)
    start = synthetic_state(grow, aggregates, largest)
    with Batch([grow], states=[start]) as b:
        b.run(max_steps=30, steps_per_launch=30)
        grown = b.store_all(raw=True)
    ends = []
    for threads in (32, 512):
        with Batch([burn], states=grown) as b:
            b.threads = threads
            b.run(max_steps=steps, steps_per_launch=steps)
            assert np.all(b.stats()["status"] == 0)
            ends.append(b.store(0))
    one, two = ends
    assert np.array_equal(one.spheres.view(np.int64), two.spheres.view(np.int64))
    assert np.array_equal(one.members, two.members) and np.array_equal(one.n_spheres, two.n_spheres)
    off, L = one.member_offsets(), one.box_length
    for a in range(one.na):
        m = one.members[off[a]:off[a + 1]]
        p, r = one.spheres[:3, m], one.spheres[S["r"], m]
        d = p[:, :, None] - p[:, None, :]
        d -= L * np.round(d / L)
        touch = (d ** 2).sum(0) <= (r[:, None] + r[None, :]) ** 2 * (1 + 1e-9) + 1e-28
        seen, todo = {0}, [0]
        while todo:
            for j in np.flatnonzero(touch[todo.pop()]):
                if j not in seen:
                    seen.add(int(j))
                    todo.append(int(j))
        assert len(seen) == len(m), a
