"""Performance cases: the work that a user of this library has it do.

Three families, all through the package's public entry points:

* contact queries on one box (``AggregatList``): one at a time as the drop-in
  loop asks them, and many at once;
* MC steps: the host-driven loop on one box (``AggregatList.calcul``) and the
  device-resident loop over many boxes (``Batch``), whole calls from states in
  page-locked host arrays to the final states back in host arrays, without and
  with surface reactions;
* the continuous-batching server (``Server``), from submitted parameters to
  final states.

Sizes are those of the benchmark's workloads (boxes of 256 to 16 384 monomers
at 100 to 5000 ppm, a 1 000 000-sphere snapshot with 10 000 queries, serving
requests from a few hundred monomers up) and of the tests (boxes of 300 to
1000 monomers, surface growth and oxidation).
"""
from __future__ import annotations

import math
import random

import numpy as np

from mcac_gb300 import (AggregatList, Batch, PhysicalModel, Server, StateBuffers, init_state, synthetic_state)
from mcac_gb300._lib import State, f64, i64, ptr
from mcac_gb300.snapshot import A, S
from mcac_gb300.workloads import random_directions

# growth fluxes in kg/m^2/s: the serving workload's, and oxidation
FLUX = {"none": 0.0, "growth": 1e-3, "individual": 1e-3, "oxidation": -0.5}


def listed() -> list[dict]:
    return [
        # contact queries one at a time, as the drop-in per-step interface asks
        # them, on the box of the basic configuration (1000 monomers as placed):
        # pure latency
        {"name": "query one by one", "kind": "query", "spheres": 1000, "aggregates": 1000, "largest": 1, "queries": 64,
         "ppm": 1000.0, "sigma": 1.0, "one_by_one": True},
        # a handful of trial moves asked at once on a middling box
        {"name": "query 64 of 20k", "kind": "query", "spheres": 20000, "aggregates": 400, "largest": 500,
         "queries": 64, "ppm": 5000.0, "sigma": 1.5, "one_by_one": False},
        # the contact-search benchmark: 10 000 queries on a million spheres
        {"name": "query 10k of 1M", "kind": "query", "spheres": 1000000, "aggregates": 20000, "largest": 500,
         "queries": 10000, "ppm": 5000.0, "sigma": 1.5, "one_by_one": False},
        # the end of a run: a dozen aggregates of more than a thousand spheres
        # each, where a query meets millions of sphere pairs
        {"name": "query 500 late", "kind": "query", "spheres": 16001, "aggregates": 12, "largest": 4000,
         "queries": 500, "ppm": 5000.0, "sigma": 1.25, "one_by_one": False},
        # the host-driven loop (step-exact with the reference) on the basic
        # configuration: one query, translation and merge per call
        {"name": "calcul 1000", "kind": "calcul", "spheres": 1000, "aggregates": 1000, "largest": 1, "steps": 500,
         "ppm": 1000.0, "sigma": 1.0, "reactions": "none"},
        # one box in the device loop, as run_device serves it
        {"name": "loop one 4096", "kind": "loop", "boxes": 1, "spheres_min": 4096, "spheres_max": 4096,
         "aggregates": 0, "largest": 1, "steps": 2000, "ppm_min": 1000.0, "ppm_max": 1000.0, "reactions": "none",
         "volsurf": "none"},
        # the benchmark ensemble's early steps: 512 boxes of 256 to 16 384 monomers
        {"name": "loop ensemble 512", "kind": "loop", "boxes": 512, "spheres_min": 256, "spheres_max": 16384,
         "aggregates": 0, "largest": 1, "steps": 4000, "ppm_min": 100.0, "ppm_max": 5000.0, "reactions": "none",
         "volsurf": "none"},
        # the same kind of boxes late in their runs: tens of large aggregates
        {"name": "loop late 152", "kind": "loop", "boxes": 152, "spheres_min": 2000, "spheres_max": 8000,
         "aggregates": 60, "largest": 600, "steps": 500, "ppm_min": 1000.0, "ppm_max": 5000.0, "reactions": "none",
         "volsurf": "none"},
        # many replicas of a small box, one warp each
        {"name": "loop replicas 2000", "kind": "loop", "boxes": 2000, "spheres_min": 1000, "spheres_max": 1000,
         "aggregates": 0, "largest": 1, "steps": 2000, "ppm_min": 1000.0, "ppm_max": 1000.0, "reactions": "none",
         "volsurf": "none"},
        # surface growth of every aggregate at every step, overlap-corrected volumes
        {"name": "loop growth 64", "kind": "loop", "boxes": 64, "spheres_min": 300, "spheres_max": 1500,
         "aggregates": 0, "largest": 1, "steps": 100, "ppm_min": 5000.0, "ppm_max": 5000.0, "reactions": "growth",
         "volsurf": "caps"},
        # oxidation: shrinking spheres, removals and splits checked every step
        {"name": "loop oxidation 16", "kind": "loop", "boxes": 16, "spheres_min": 300, "spheres_max": 1500,
         "aggregates": 15, "largest": 300, "steps": 40, "ppm_min": 5000.0, "ppm_max": 5000.0,
         "reactions": "oxidation", "volsurf": "none"},
        # a burst of serving requests, each to an eighth of its monomers' number
        {"name": "serve 48", "kind": "serve", "requests": 48, "capacity": 32, "spheres_min": 300,
         "spheres_max": 1500, "epoch": 5000, "growing": 0.0},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["query", "query", "calcul", "loop", "loop", "loop", "reactions", "serve"])
    if kind == "query":
        n = int(_log(rng, 500, 1000000))
        late = rng.random() < 0.3
        na = rng.randint(8, 60) if late else max(2, int(n / _log(rng, 1.5, 80)))
        n = min(n, 30000) if late else n
        largest = 4000 if late else 500
        return {"kind": "query", "spheres": n, "aggregates": na, "largest": largest,
                "queries": int(_log(rng, 64, 500 if late else 10000)), "ppm": _log(rng, 300, 5000),
                "sigma": rng.choice([1.0, 1.25, 1.5]), "one_by_one": rng.random() < 0.25}
    if kind == "calcul":
        n = int(_log(rng, 300, 8000))
        placed = rng.random() < 0.5
        return {"kind": "calcul", "spheres": n, "aggregates": n if placed else max(2, n // 20),
                "largest": 1 if placed else 400, "steps": rng.randint(100, 500), "ppm": _log(rng, 300, 5000),
                "sigma": rng.choice([1.0, 1.25]), "reactions": "none"}
    if kind == "loop":
        boxes = int(_log(rng, 1, 2000))
        top = int(min(16384, _log(rng, 600, max(700, 2.5e6 / boxes))))
        late = rng.random() < 0.4
        lo = int(_log(rng, 256, 0.8 * top))
        if late:
            top, lo = min(top, 8000), min(lo, 6000)
        return {"kind": "loop", "boxes": min(boxes, 600) if late else boxes, "spheres_min": lo, "spheres_max": top,
                "aggregates": rng.randint(12, 120) if late else 0, "largest": 600 if late else 1,
                "steps": rng.randint(100, 400) if late else rng.randint(200, 1500), "ppm_min": 300.0,
                "ppm_max": _log(rng, 1000, 5000), "reactions": "none", "volsurf": "none"}
    if kind == "reactions":
        how = rng.choice(["growth", "individual", "oxidation"])
        top = int(_log(rng, 350, 1500))
        return {"kind": "loop", "boxes": int(_log(rng, 1, 64 if how != "oxidation" else 16)), "spheres_min": 300,
                "spheres_max": top, "aggregates": 0 if how != "oxidation" else rng.randint(8, 20),
                "largest": 1 if how != "oxidation" else 300, "steps": rng.randint(20, 100 if how != "oxidation" else 40),
                "ppm_min": 1000.0, "ppm_max": 5000.0, "reactions": how,
                "volsurf": "none" if how == "oxidation" else rng.choice(["none", "caps", "alphas"])}
    return {"kind": "serve", "requests": int(_log(rng, 4, 48)), "capacity": rng.choice([8, 16, 32]), "spheres_min": 300,
            "spheres_max": int(_log(rng, 400, 1500)), "epoch": rng.randint(2000, 8000), "growing": 0.0}


# ------------------------------------------------------------------ inputs
def _ini(n: int, seed: int, ppm: float, sigma: float, reactions: str = "none", volsurf: str = "none",
         limit: int = 1) -> str:
    surface = ""
    if reactions != "none":
        surface = (f"[surface_growth]\nwith_surface_reactions = true\nflux_surfgrowth = {FLUX[reactions]!r}\n"
                   f"volsurf_method = {volsurf}\nfull_aggregate_update_frequency = 1\n[oxidation]\nrp_min = 2e-9\n")
    return (f"[monomers]\nnumber = {n}\ndensity = 1800\nmean_diameter = 30\ndispersion_diameter = {sigma!r}\n"
            f"initialisation_mode = lognormal\n[environment]\nvolume_fraction = {ppm * 1e-6!r}\n"
            f"temperature = 1700\npressure = 101300\nfractal_prefactor = 1.4\nfractal_dimension = 1.8\n{surface}"
            f"[limits]\nnumber_of_aggregates = {limit}\nn_iter_without_event = 10000\n"
            f"[numerics]\nrandom_seed = {seed}\nwith_domain_duplication = false\n"
            + ("individual_surf_reactions = true\n" if reactions == "individual" else ""))


class Arrays:
    """The states of many boxes in five page-locked arrays, one box behind the
    other, with a StateBuffers of views for each box."""

    def __init__(self, sizes: list[tuple[int, int]]):
        ns, na = sum(s for s, _ in sizes), sum(a for _, a in sizes)
        # one page-locked block, zeroed
        block = StateBuffers(ns, na, pinned=True)
        self.fields = {k: getattr(block, k) for k in ("spheres", "sphere_label", "aggregates", "n_spheres", "members")}
        for v in self.fields.values():
            v[...] = 0
        self.fields["spheres"] = self.fields["spheres"].reshape(-1)
        self.fields["aggregates"] = self.fields["aggregates"].reshape(-1)
        self.boxes = []
        s0 = a0 = 0
        for s, a in sizes:
            b = StateBuffers(1, 1)
            b.spheres = self.fields["spheres"][9 * s0:9 * (s0 + s)].reshape(9, s)
            b.sphere_label = self.fields["sphere_label"][s0:s0 + s]
            b.aggregates = self.fields["aggregates"][21 * a0:21 * (a0 + a)].reshape(21, a)
            b.n_spheres = self.fields["n_spheres"][a0:a0 + a]
            b.members = self.fields["members"][s0:s0 + s]
            b.state = State(s, a, 0, 0.0, 0.0, 0.0, ptr(b.spheres, f64), ptr(b.sphere_label, i64),
                            ptr(b.aggregates, f64), ptr(b.n_spheres, i64), ptr(b.members, i64))
            self.boxes.append(b)
            s0, a0 = s0 + s, a0 + a

    def put(self, k: int, src: StateBuffers) -> None:
        b, st = self.boxes[k], src.state
        ns, na = int(st.n_spheres), int(st.n_aggregates)
        b.spheres[...] = src.spheres.reshape(-1)[:9 * ns].reshape(9, ns)
        b.sphere_label[...] = src.sphere_label[:ns]
        b.aggregates[...] = src.aggregates.reshape(-1)[:21 * na].reshape(21, na)
        b.n_spheres[...] = src.n_spheres[:na]
        b.members[...] = src.members[:ns]
        for f in ("n_verlet_divisions", "box_length", "maxradius", "time"):
            setattr(b.state, f, getattr(st, f))


def _state(model: PhysicalModel, aggregates: int, largest: int) -> StateBuffers:
    n = int(model.params.n_monomeres)
    if largest == 1:
        return init_state(model)
    return synthetic_state(model, min(aggregates, n), max(largest, -(-n // aggregates)))


def _sizes(case: dict, n: int) -> list[int]:
    """n monomer numbers spread evenly over the logarithm of the case's range,
    in a scattered order."""
    lo, hi = math.log(case["spheres_min"]), math.log(case["spheres_max"])
    return [int(round(math.exp(lo + (hi - lo) * ((0.5 + 0.618033988749895 * k) % 1.0)))) for k in range(n)]


def _loop_models(case: dict, seed: int) -> list[PhysicalModel]:
    rng = np.random.Generator(np.random.PCG64([seed, 7]))
    models = []
    for k, n in enumerate(_sizes(case, case["boxes"])):
        sigma = 1.0 if rng.random() < 0.5 else 1.25
        ppm = rng.uniform(case["ppm_min"], case["ppm_max"])
        models.append(PhysicalModel(text=_ini(n, 2003 * (seed % 100000) + k + 1, ppm, sigma, case["reactions"],
                                              case["volsurf"], 0 if case["reactions"] == "oxidation" else 1)))
    return models


def _loop_inputs(case: dict, seed: int, models: list[PhysicalModel]) -> Arrays:
    if case["largest"] == 1:  # as placed: the batch places its boxes in parallel
        with Batch(models) as b:
            arrays = Arrays([b.box_sizes(k) for k in range(len(models))])
            b.store_all(raw=True, out=arrays.boxes)
        return arrays
    states = [_state(m, case["aggregates"], case["largest"]) for m in models]
    if case["reactions"] == "oxidation":
        # aggregates whose spheres overlap, as growth leaves them: a short run
        # at a high growth rate first
        grown = []
        for m in models:
            g = PhysicalModel(text=m.to_ini())
            g.set(flux_surfgrowth=4.0)
            grown.append(g)
        with Batch(grown, states=states) as b:
            b.run(max_steps=40, steps_per_launch=40)
            states = b.store_all(raw=True)
    arrays = Arrays([(int(s.state.n_spheres), int(s.state.n_aggregates)) for s in states])
    for k, s in enumerate(states):
        arrays.put(k, s)
    return arrays


def _query_inputs(case: dict, seed: int) -> dict:
    model = PhysicalModel(text=_ini(case["spheres"], seed % 2000000000, case["ppm"], case["sigma"]))
    state = _state(model, case["aggregates"], case["largest"])
    rng = np.random.Generator(np.random.PCG64([seed, 3]))
    sources = rng.integers(0, int(state.state.n_aggregates), case["queries"]).astype(np.int64)
    directions = random_directions(rng, case["queries"])
    return {"model": model, "state": state, "sources": sources, "directions": directions,
            "distances": state.aggregates[A["lpm"], sources].copy()}


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "query":
        st = _query_inputs(case, seed)
        # the box stays on the GPU, as a program that asks many queries keeps it
        st["box"] = AggregatList(st["model"], st["state"])
        st["one_by_one"] = case["one_by_one"]
    elif kind == "calcul":
        model = PhysicalModel(text=_ini(case["spheres"], seed % 2000000000, case["ppm"], case["sigma"],
                                        case["reactions"]))
        st = {"model": model, "state": _state(model, case["aggregates"], case["largest"]), "steps": case["steps"]}
    elif kind == "loop":
        models = _loop_models(case, seed)
        arrays = _loop_inputs(case, seed, models)
        room = [(b.spheres.shape[1], b.spheres.shape[1] if case["reactions"] == "oxidation" else b.aggregates.shape[1])
                for b in arrays.boxes]
        st = {"models": models, "in": arrays, "out": Arrays(room), "steps": case["steps"]}
    else:
        rng = np.random.Generator(np.random.PCG64([seed, 11]))
        models = []
        for k, n in enumerate(_sizes(case, case["requests"])):
            models.append(PhysicalModel(text=_ini(n, 2003 * (seed % 100000) + k + 1, rng.uniform(1000, 5000),
                                                  rng.uniform(1.1, 1.4), limit=max(1, n // 8))))
        st = {"models": models, "capacity": case["capacity"], "epoch": case["epoch"]}
    st["kind"] = kind
    return st


# -------------------------------------------------------------------- runs
def _run_query(st: dict) -> dict:
    box = st["box"]
    if st["one_by_one"]:
        got = [box.distance_to_next_contact(int(s), d, float(t))
               for s, d, t in zip(st["sources"], st["directions"], st["distances"])]
        return {"distance": np.array([g.distance for g in got]),
                "moving_sphere": np.array([g.moving_sphere for g in got]),
                "moving_aggregate": np.array([g.moving_aggregate for g in got]),
                "other_sphere": np.array([g.other_sphere for g in got]),
                "other_aggregate": np.array([g.other_aggregate for g in got])}
    out, _ = box.distance_to_next_contacts(st["sources"], st["directions"], st["distances"])
    return {k: out[k] for k in ("distance", "moving_sphere", "moving_aggregate", "other_sphere", "other_aggregate")}


def _table(rows: np.ndarray, n: int) -> np.ndarray:
    """A final table with as many columns as there were aggregates to begin
    with (how many are left is the run's result)."""
    out = np.zeros(rows.shape[:-1] + (n,), dtype=rows.dtype)
    out[..., :rows.shape[-1]] = rows
    return out


def _run_calcul(st: dict) -> dict:
    with AggregatList(st["model"], st["state"]) as box:
        stats, _ = box.calcul(max_steps=st["steps"])
        final = box.store()
    n = len(st["state"].n_spheres)
    return {"spheres": final.spheres, "sphere_label": final.sphere_label, "aggregates": _table(final.aggregates, n),
            "n_spheres": _table(final.n_spheres, n), "members": final.members, "time": final.time,
            "steps": int(stats.steps), "events": int(stats.events)}


def _run_loop(st: dict) -> dict:
    with Batch(st["models"], states=st["in"].boxes) as batch:
        batch.run(max_steps=st["steps"], steps_per_launch=st["steps"])
        stats = batch.stats()
        batch.store_all(raw=True, out=st["out"].boxes)
    return dict(st["out"].fields, **{f: stats[f] for f in ("steps", "events", "n_aggregates", "time", "status")})


def _run_serve(st: dict) -> dict:
    with Server(st["capacity"], keep_final_states=True) as server:
        server.set_threads(0)
        ids = [server.submit(m) for m in st["models"]]
        done = []
        while True:
            active, pending = server.step(st["epoch"])
            done.append(server.poll())
            if active == 0 and pending == 0:
                break
        finals = [server.final_state(i) for i in ids]
    done = np.concatenate(done)
    done = done[np.argsort(done["id"])]
    out = {f: done[f] for f in ("id", "steps", "events", "n_aggregates", "time", "status", "finished")}
    out["spheres"] = np.concatenate([s.spheres.reshape(-1) for s in finals])
    out["aggregates"] = np.concatenate([_table(s.aggregates, s.ns).reshape(-1) for s in finals])
    out["n_spheres"] = np.concatenate([_table(s.n_spheres, s.ns) for s in finals])
    for f in ("sphere_label", "members"):
        out[f] = np.concatenate([getattr(s, f) for s in finals])
    return out


def run(state: dict):
    return {"query": _run_query, "calcul": _run_calcul, "loop": _run_loop, "serve": _run_serve}[state["kind"]](state)


def work(case: dict) -> dict:
    """Bytes: inputs once, outputs once. Flops: what the sphere and aggregate
    tests that no search structure can avoid cost (tens of operations each)."""
    if case["kind"] == "query":
        q, per = case["queries"], case["spheres"] / case["aggregates"]
        # a query's own inputs and result, and the spheres of its aggregate
        return {"bytes": q * (40 + 40 + 16 * per) + min(q * 32, case["aggregates"] * 32), "flops": q * 50 * (per + 20)}
    if case["kind"] == "calcul":
        ns, na, steps = case["spheres"], case["aggregates"], case["steps"]
        return {"bytes": 2 * (88 * ns + 176 * na) + steps * 500, "flops": steps * 2000}
    if case["kind"] == "loop":
        mean = (case["spheres_max"] - case["spheres_min"]) / math.log(case["spheres_max"] / case["spheres_min"]) \
            if case["spheres_max"] > case["spheres_min"] else case["spheres_min"]
        na = case["aggregates"] or mean
        per_step = 2000 if case["reactions"] == "none" else 2000 + 60 * mean
        return {"bytes": case["boxes"] * 2 * (88 * mean + 176 * na),
                "flops": case["boxes"] * case["steps"] * per_step}
    mean = (case["spheres_max"] - case["spheres_min"]) / math.log(case["spheres_max"] / case["spheres_min"])
    return {"bytes": case["requests"] * mean * (88 + 176 / 8), "flops": case["requests"] * mean * 20 * 2000}


# ------------------------------------------------------------------- exact
def _wrap(d, L):
    return d - L * np.round(d / L)


def _exact_distances(case: dict, seed: int) -> np.ndarray:
    """The least swept distance of each query over every sphere of the other
    aggregates, 0 for spheres that touch already, infinity without a contact."""
    st = _query_inputs(case, seed)
    sb, L = st["state"], float(st["state"].state.box_length)
    pos = sb.spheres[[S["x"], S["y"], S["z"]]].T
    rad = sb.spheres[S["r"]]
    centre = sb.aggregates[[A["x"], A["y"], A["z"]]].T
    count, members = sb.n_spheres, sb.members
    off = np.concatenate([[0], np.cumsum(count)])
    owner = np.repeat(np.arange(len(count)), count)
    reach = np.zeros(len(count))  # from the aggregate's centre to its outermost point
    np.maximum.at(reach, owner, np.sqrt((_wrap(pos[members] - centre[owner], L) ** 2).sum(1)) + rad[members])
    # aggregates by cells wider than any query's reach, when the box holds a few
    G = max(1, int(L / (2.001 * reach.max() + st["distances"].max())))
    G = min(G, 32) if G >= 4 else 1
    cell = np.floor(centre / L * G).astype(np.int64) % G
    ident = (cell[:, 0] * G + cell[:, 1]) * G + cell[:, 2]
    order = np.argsort(ident, kind="stable")
    start = np.searchsorted(ident[order], np.arange(G ** 3 + 1))
    step = np.stack(np.meshgrid(*[np.arange(-1, 2)] * 3, indexing="ij"), -1).reshape(-1, 3) if G > 1 else np.zeros((1, 3), int)
    out = np.full(case["queries"], np.inf)
    for q in range(case["queries"]):
        a, u, t = int(st["sources"][q]), st["directions"][q], float(st["distances"][q])
        c = (cell[a] + step) % G
        c = (c[:, 0] * G + c[:, 1]) * G + c[:, 2]
        some = np.concatenate([order[start[k]:start[k + 1]] for k in c])
        some = some[some != a]
        d = _wrap(centre[some] - centre[a] - 0.5 * t * u, L) + 0.5 * t * u
        along = np.clip(d @ u, 0.0, t)
        near = np.sqrt(((d - along[:, None] * u) ** 2).sum(1)) <= (reach[some] + reach[a]) * (1 + 1e-9)
        cand = some[near]
        if not len(cand):
            continue
        mine = members[off[a]:off[a + 1]]
        for c in cand:
            other = members[off[c]:off[c + 1]]
            for i0 in range(0, len(mine), 512):
                m = mine[i0:i0 + 512]
                e = pos[other][None, :, :] - pos[m][:, None, :]
                e = _wrap(e - 0.5 * t * u, L) + 0.5 * t * u
                s2 = (rad[m][:, None] + rad[other][None, :]) ** 2
                proj = e @ u
                d2 = (e ** 2).sum(2)
                axis = (np.cross(e, u) ** 2).sum(2)
                end = ((e - t * u) ** 2).sum(2) <= s2
                hit = (proj >= 0) & (end | (proj <= t)) & (axis <= s2)
                v = np.where(hit, proj - np.sqrt(np.maximum(s2 - axis, 0.0)), np.inf)
                v = np.where((_wrap(e, L) ** 2).sum(2) <= s2, 0.0, v)
                out[q] = min(out[q], v.min())
    return out


def exact(case: dict, seed: int):
    # runs are chains of random moves, each decided by the rounding of the
    # ones before it: no value of them can be had in another arithmetic
    if case["kind"] != "query":
        return None
    pairs = case["queries"] * (case["spheres"] / case["aggregates"]) ** 2 * (2 if case["largest"] <= 500 else 10)
    if pairs > 1e8:
        return None
    return {"distance": _exact_distances(case, seed), "moving_sphere": None, "moving_aggregate": None,
            "other_sphere": None, "other_aggregate": None}
