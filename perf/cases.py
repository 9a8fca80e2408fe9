"""Performance cases of the pair-distance and histogram path.

Each case is one pass of work that a fit does through the package's public
entry points, with the inputs a program has in hand before the call:

* ``move``: ``multiple_pairs_histograms_coords`` of the moved atoms, which a
  PairDistributionConstraint calls before and after every move;
* ``full``: ``full_pairs_histograms_coords``, the all-pairs histogram of a
  constraint's compute_data;
* ``contacts``: ``atomic_distances`` of InterMolecularDistanceConstraint, for
  a moved molecule or for all atoms;
* ``coordination``: ``atomic_coordination`` of
  AtomicCoordinationNumberConstraint, for a moved molecule or for all atoms;
* ``distances``: ``pairs_distances`` rows of some atoms to all atoms;
* ``sine``: the FP64 transforms between real and reciprocal space;
* ``shape``: the ShapeFunction of a finite cluster (no periodic box);
* ``batch``: batched Metropolis steps of many engines from host arrays;
* ``chain``: steps of one resident engine, single atoms or whole molecules;
* ``serve``: iterations of a serving loop over live fits with an S(Q) term.

The drop-in calls take and return host arrays, as fullrmc's constraints use
them; the engines keep their state on the device between passes.
"""
import math

import numpy as np
import torch

from fullrmc_gb300 import (atomic_coordination, atomic_distances, pairs_distances, pairs_histograms,
                           reciprocal_space, shape_function, synthetic)
from fullrmc_gb300.engine import EngineSet, group_moves, translation_moves

F32 = np.float32
RING = 13   # atoms of one ring molecule (synthetic.ring_molecules)


def listed():
    return [
        # the smallest call of a fit: one moved atom of a 5,000-atom binary alloy (latency)
        {"name": "move_alloy_5000", "kind": "move", "n": 5000, "ne": 2, "box": "cubic", "k": 1, "rmax": 15.0},
        # a moved 13-atom ring of a 52,000-atom molecular system
        {"name": "move_ring_52000", "kind": "move", "n": 52000, "ne": 3, "box": "rings", "k": 13, "rmax": 15.0},
        # start-up histogram of the largest configuration: 5e9 pairs, triclinic gamma = 120
        {"name": "full_triclinic_100000", "kind": "full", "n": 100000, "ne": 3, "box": "hexagonal", "rmax": 20.0},
        # start-up histogram of an ordinary engine: odd size, four elements, general triclinic box
        {"name": "full_triclinic_11303", "kind": "full", "n": 11303, "ne": 4, "box": "triclinic", "rmax": 12.0},
        # start-up of an intermolecular distance constraint on 1,538 rings
        {"name": "contacts_all_19994", "kind": "contacts", "nmol": 1538, "rows": "all", "reduce": "upper"},
        # start-up of a coordination-number constraint with four definitions on 4,000 rings
        {"name": "coordination_all_52000", "kind": "coordination", "nmol": 4000, "rows": "all"},
        # distance rows of a moved ring to all atoms
        {"name": "distances_13x52000", "kind": "distances", "n": 52000, "box": "cubic", "k": 13},
        # G(r) to S(Q) on the largest grids: r 0-20 by 0.01, Q 0.5-30 by 0.01
        {"name": "sine_2001x2951", "kind": "sine", "way": "Gr_to_sq", "nr": 2001, "nq": 2951},
        # shape function of a 100,000-atom particle, every pair counted
        {"name": "shape_cluster_100000", "kind": "shape", "n": 100000, "ne": 3, "dr": 1.0},
        # many independent fits side by side, moves from the host every step
        {"name": "batch_256_engines", "kind": "batch", "engines": 256, "nmin": 1000, "nmax": 20000, "steps": 16},
        # one fit alone with molecule moves (translations and rotations)
        {"name": "chain_rings_52000", "kind": "chain", "n": 52000, "box": "rings", "rmax": 15.0, "steps": 64},
        # a serving loop's live fits, each with G(r) and S(Q)
        {"name": "serve_24_fits", "kind": "serve", "fits": 24, "nmin": 2000, "nmax": 200000, "steps": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["move", "full", "contacts", "coordination", "distances", "sine", "shape", "batch", "chain",
                       "serve"])
    box = rng.choice(["cubic", "hexagonal", "triclinic"])
    if kind == "move":
        if rng.random() < 0.5:
            return {"kind": kind, "n": RING * _log(rng, 80, 8000), "ne": 3, "box": "rings", "k": RING,
                    "rmax": round(rng.uniform(10, 20), 1)}
        return {"kind": kind, "n": _log(rng, 1000, 200000), "ne": rng.randint(1, 4), "box": box,
                "k": rng.choice([1, 1, 2, 5, 13]), "rmax": round(rng.uniform(8, 20), 1)}
    if kind == "full":
        return {"kind": kind, "n": _log(rng, 1000, 100000), "ne": rng.randint(1, 4), "box": box,
                "rmax": round(rng.uniform(8, 20), 1)}
    if kind == "contacts":
        return {"kind": kind, "nmol": _log(rng, 80, 1538), "rows": rng.choice(["all", "molecule"]),
                "reduce": rng.choice(["none", "upper", "nearest"])}
    if kind == "coordination":
        return {"kind": kind, "nmol": _log(rng, 80, 4000), "rows": rng.choice(["all", "molecule"])}
    if kind == "distances":
        return {"kind": kind, "n": _log(rng, 1000, 200000), "box": box, "k": rng.choice([1, 1, 5, 13])}
    if kind == "sine":
        return {"kind": kind, "way": rng.choice(["Gr_to_sq", "gr_to_sq", "sq_to_Gr"]), "nr": rng.randint(501, 2001),
                "nq": rng.randint(451, 2951)}
    if kind == "shape":
        return {"kind": kind, "n": _log(rng, 5000, 100000), "ne": rng.randint(1, 4),
                "dr": rng.choice([0.5, 1.0, 2.0])}
    if kind == "batch":
        return {"kind": kind, "engines": _log(rng, 8, 256), "nmin": 1000, "nmax": _log(rng, 2000, 20000),
                "steps": 16}
    if kind == "chain":
        if rng.random() < 0.4:
            return {"kind": kind, "n": RING * _log(rng, 200, 4000), "box": "rings",
                    "rmax": round(rng.uniform(10, 15), 1), "steps": 64}
        return {"kind": kind, "n": _log(rng, 2000, 100000), "box": box, "rmax": round(rng.uniform(10, 20), 1),
                "steps": 64}
    return {"kind": kind, "fits": rng.randint(4, 24), "nmin": 2000, "nmax": _log(rng, 5000, 200000), "steps": 64}


# ------------------------------------------------------------------ inputs
def _basis(box, n, rho=0.1):
    unit = {"cubic": np.eye(3), "hexagonal": synthetic.triclinic(1.0, 1.0, 1.0, 90, 90, 120),
            "triclinic": synthetic.triclinic(1.0, 1.1, 0.9, 85, 97, 112)}[box].astype(np.float64)
    a = (n / rho / abs(np.linalg.det(unit))) ** (1.0 / 3.0)
    return (unit * a).astype(F32)


def _system(case, seed):
    """One system: uniform coordinates in the box, or randomly placed rings."""
    if case["box"] == "rings":
        return synthetic.ring_molecules(seed=seed, nmol=case["n"] // RING, rmax=case["rmax"])
    rng = np.random.default_rng([seed, 1])
    fr = rng.dirichlet(np.full(case.get("ne", 2), 8.0))
    return synthetic.make_system(rng, case["n"], fr, _basis(case["box"], case["n"]), case["rmax"])


def _hist_args(s):
    m = s.model
    return dict(boxCoords=s.box_coords, basis=s.basis, isPBC=True, moleculeIndex=s.mol.astype(np.int32),
                elementIndex=s.el.astype(np.int32), numberOfElements=len(m.elements_count),
                minDistance=F32(m.minDistance), maxDistance=F32(m.maxDistance), bin=F32(m.bin), histSize=int(m.hs))


def _moved(case, seed, n):
    rng = np.random.default_rng([seed, 2])
    if case["box"] == "rings":
        return np.arange(RING, dtype=np.int32) + RING * int(rng.integers(0, n // RING))
    return np.sort(rng.choice(n, case["k"], replace=False)).astype(np.int32)


def _contacts_args(case, seed):
    s = synthetic.ring_molecules(seed=seed, nmol=case["nmol"])
    rng = np.random.default_rng([seed, 3])
    lo = np.zeros((3, 3, 1), F32)
    up = rng.uniform(1.8, 2.6, (3, 3))
    up = ((up + up.T) / 2).astype(F32).reshape(3, 3, 1)
    kw = dict(boxCoords=s.box_coords, basis=s.basis, isPBC=True, moleculeIndex=s.mol, elementIndex=s.el,
              numberOfElements=3, lowerLimit=lo, upperLimit=up, intraMolecular=False, countWithinLimits=True,
              reduceDistanceToUpper=case["reduce"] == "upper", reduceDistance=case["reduce"] == "nearest")
    if case["rows"] == "molecule":
        kw["indexes"] = np.arange(RING, dtype=np.int32) + RING * int(rng.integers(0, case["nmol"]))
    return kw


# (core element, shell element, lower, upper): C-O both ways, C-H and C-C bonds
_DEFINITIONS = ((0, 1, 1.0, 1.6), (1, 0, 1.0, 1.6), (0, 2, 0.9, 1.3), (0, 0, 1.2, 1.6))


def _coordination_args(case, seed):
    """The lists AtomicCoordinationNumberConstraint builds from its definitions."""
    s = synthetic.ring_molecules(seed=seed, nmol=case["nmol"])
    n = s.box_coords.shape[0]
    core, shell = [[] for _ in range(n)], [[] for _ in range(n)]
    cores = [np.flatnonzero(s.el == d[0]).astype(np.int32) for d in _DEFINITIONS]
    shells = [np.flatnonzero(s.el == d[1]).astype(np.int32) for d in _DEFINITIONS]
    for d in range(len(_DEFINITIONS)):
        for a in cores[d]:
            core[a].append(d)
        for a in shells[d]:
            shell[a].append(d)
    kw = dict(boxCoords=s.box_coords, basis=s.basis, isPBC=True, coresIndexes=cores, shellsIndexes=shells,
              lowerShells=[F32(d[2]) for d in _DEFINITIONS], upperShells=[F32(d[3]) for d in _DEFINITIONS],
              asCoreDefIdxs=[np.array(x, np.int32) for x in core],
              inShellDefIdxs=[np.array(x, np.int32) for x in shell])
    if case["rows"] == "molecule":
        first = RING * int(np.random.default_rng([seed, 4]).integers(0, case["nmol"]))
        kw["indexes"] = np.arange(first, first + RING, dtype=np.int32)
    return kw


def _sine_args(case, seed):
    rng = np.random.default_rng([seed, 5])
    r = (0.01 * np.arange(case["nr"])).astype(F32)
    q = (0.5 + 0.01 * np.arange(case["nq"])).astype(F32)
    G = synthetic.synthetic_G(rng, r, 0.1)
    if case["way"] == "Gr_to_sq":
        return dict(distances=r, Gr=G, qrange=q)
    if case["way"] == "gr_to_sq":
        g = (1.0 + G.astype(np.float64) / (4 * np.pi * 0.1 * np.maximum(r, 0.01).astype(np.float64))).astype(F32)
        return dict(distances=r, gr=g, qrange=q, rho=0.1)
    S = (1.0 + np.exp(-0.1 * q.astype(np.float64)) * np.sin(2.5 * q.astype(np.float64)) +
         rng.normal(0.0, 0.01, q.shape)).astype(F32)
    return dict(qValues=q, rValues=r, sq=S)


def _shape_args(case, seed):
    """A spherical particle of uniform density 0.1 atoms/A^3 in free space."""
    rng = np.random.default_rng([seed, 6])
    n = case["n"]
    radius = (3.0 * n / (4.0 * np.pi * 0.1)) ** (1.0 / 3.0)
    v = rng.normal(size=(n, 3))
    v *= (radius * rng.random(n) ** (1.0 / 3.0) / np.linalg.norm(v, axis=1))[:, None]
    el = rng.integers(0, case["ne"], size=n).astype(np.int32)
    return dict(boxCoords=v.astype(F32), basis=np.eye(3, dtype=F32), isPBC=False,
                moleculeIndex=np.arange(n, dtype=np.int32), elementIndex=el,
                elementsCount=np.bincount(el, minlength=case["ne"]), weights=[6.0, 8.0, 14.0, 26.0][:case["ne"]],
                volume=4.0 / 3.0 * np.pi * radius ** 3, rValues=(0.005 + 0.01 * np.arange(2000)).astype(F32),
                qmin=0.001, qmax=1.0, dq=0.005, rmin=0.0, rmax=float(math.ceil(2.2 * radius)), dr=case["dr"])


def _engine_systems(case, seed):
    if case["kind"] == "batch":
        return synthetic.mixed_engines(seed=seed, count=case["engines"], nmin=case["nmin"], nmax=case["nmax"])
    if case["kind"] == "serve":
        return [synthetic.serving_fit(100 * seed + k, nmin=case["nmin"], nmax=case["nmax"])[0]
                for k in range(case["fits"])]
    return [_system(case, seed)]


_STREAM = 4096  # moves of an engine's stream; a longer run starts over


def _streams(case, systems, seed):
    if case["kind"] == "chain" and case["box"] == "rings":
        return [group_moves(np.random.default_rng([seed, 7]), systems[0].groups, 1024, 0.1, 10.0)]
    return [translation_moves(np.random.default_rng([seed, 7, e]), s.box_coords.shape[0], _STREAM, 0.1)
            for e, s in enumerate(systems)]


class _Engines:
    """A program's handle on its engines: the set, the moves ahead and how far it is."""

    def __init__(self, case, seed):
        self.systems = _engine_systems(case, seed)
        self.moves = _streams(case, self.systems, seed)
        self.steps = case["steps"]
        self.done = self.pushed = 0
        if case["kind"] == "serve":
            self.es = EngineSet([], move_cap=_STREAM, tune=(1024, 512, 1))
            self.ids = [self.es.add(s) for s in self.systems]
        else:
            self.es = EngineSet(self.systems, move_cap=_STREAM)
            self.es.init()
            self.ids = list(range(len(self.systems)))
        if case["kind"] == "batch":
            # host moves per step: (steps of the stream, engines)
            self.atoms = np.ascontiguousarray(np.stack([m[0] for m in self.moves], axis=1))
            self.vecs = np.ascontiguousarray(np.stack([m[1] for m in self.moves], axis=1))
            self.u = np.ascontiguousarray(np.stack([m[2] for m in self.moves], axis=1))

    def refill(self, push):
        """Tops up the move rings when fewer moves than a pass are ahead."""
        if self.pushed - self.done >= self.steps:
            return
        length = len(self.moves[0][-1])
        for e, m in zip(self.ids, self.moves):
            push(e, *m, self.pushed)
        self.pushed += length


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("move", "full"):
        s = _system(case, seed)
        args = _hist_args(s)
        if kind == "move":
            args["indexes"] = _moved(case, seed, s.box_coords.shape[0])
        return kind, args
    if kind == "contacts":
        return kind, _contacts_args(case, seed)
    if kind == "coordination":
        return kind, _coordination_args(case, seed)
    if kind == "distances":
        rng = np.random.default_rng([seed, 8])
        return kind, dict(indexes=np.sort(rng.choice(case["n"], case["k"], replace=False)).astype(np.int32),
                          coords=rng.random((case["n"], 3)).astype(F32), basis=_basis(case["box"], case["n"]),
                          isPBC=True)
    if kind == "sine":
        return kind, (case["way"], _sine_args(case, seed))
    if kind == "shape":
        return kind, _shape_args(case, seed)
    return kind, _Engines(case, seed)


# --------------------------------------------------------------------- run
def _run_batch(p):
    """Host steps, two in flight: submit step k + 1 before step k is collected."""
    c2 = np.empty((p.steps, len(p.ids)))
    acc = np.empty((p.steps, len(p.ids)), np.int32)
    for k in range(p.steps):
        at = (p.done + k) % _STREAM
        p.es.step_host_submit(p.atoms[at], p.vecs[at], p.u[at], k & 1)
        if k:
            p.es.step_host_collect((k - 1) & 1, (c2[k - 1], acc[k - 1]))
    p.es.step_host_collect((p.steps - 1) & 1, (c2[p.steps - 1], acc[p.steps - 1]))
    p.done += p.steps
    return c2, acc


def _run_chain(p):
    p.refill(p.es.push_group_moves if p.systems[0].group_size > 1 else p.es.push_moves)
    p.es.step(p.steps, engine=p.ids[0], graph=True)
    c2, acc, atoms = p.es.results(p.ids[0], p.done, p.steps)
    p.done += p.steps
    return c2, acc, atoms


def _run_serve(p):
    p.refill(p.es.push_moves)
    for _ in range(p.steps // 32):
        p.es.step(32, graph=True)
    out = [p.es.results(e, p.done, p.steps) for e in p.ids]
    p.done += p.steps
    return np.stack([o[0] for o in out]), np.stack([o[1] for o in out])


def run(state):
    kind, a = state
    if kind == "move":
        return pairs_histograms.multiple_pairs_histograms_coords(**a)
    if kind == "full":
        return pairs_histograms.full_pairs_histograms_coords(**a)
    if kind == "contacts":
        return (atomic_distances.multiple_atomic_distances_coords if "indexes" in a else
                atomic_distances.full_atomic_distances_coords)(**a)
    if kind == "coordination":
        data = np.zeros(len(_DEFINITIONS), F32)
        (atomic_coordination.multi_atoms_coord_number_coords if "indexes" in a else
         atomic_coordination.all_atoms_coord_number_coords)(coordNumData=data, **a)
        return data
    if kind == "distances":
        return pairs_distances.pairs_distances_to_multi_indexcoords(**a)
    if kind == "sine":
        return getattr(reciprocal_space, a[0])(**a[1])
    if kind == "shape":
        Gs, more = shape_function.gr_shape_function(details=True, **a)
        return Gs, more["Gr"], more["Sq"]
    return {"batch": _run_batch, "chain": _run_chain, "serve": _run_serve}[kind](a)


# -------------------------------------------------------------------- work
def _in_range(n, rmax, rho=0.1):
    return n * min(n, 4.0 / 3.0 * math.pi * rmax ** 3 * rho)


def work(case):
    """Inputs read once, outputs written once; flops: 25 of a minimum-image distance for each pair in range."""
    kind = case["kind"]
    if kind in ("move", "full"):
        hist = 8.0 * case["ne"] ** 2 * (case["rmax"] * 100 + 1)
        rows = case["k"] if kind == "move" else case["n"] / 2
        return {"bytes": 20.0 * case["n"] + hist, "flops": 25.0 * _in_range(case["n"], case["rmax"]) / case["n"] * rows}
    if kind in ("contacts", "coordination"):
        n = RING * case["nmol"]
        rows = n / 2 if case["rows"] == "all" else RING
        near = 2.6 if kind == "contacts" else 1.6
        return {"bytes": 20.0 * n + (8.0 * n if kind == "coordination" else 0.0),
                "flops": 25.0 * _in_range(n, near) / n * rows}
    if kind == "distances":
        return {"bytes": 12.0 * case["n"] + 4.0 * case["n"] * case["k"], "flops": 25.0 * case["n"] * case["k"]}
    if kind == "sine":
        return {"bytes": 12.0 * (case["nr"] + case["nq"]), "flops": 20.0 * case["nr"] * case["nq"]}
    if kind == "shape":
        return {"bytes": 20.0 * case["n"], "flops": 12.5 * case["n"] * (case["n"] - 1.0)}
    if kind == "chain":
        atoms, rows = case["n"], RING if case["box"] == "rings" else 1
        systems, near = 1, min(1.0, 4.0 / 3.0 * math.pi * case["rmax"] ** 3 * 0.1 / case["n"])
    else:
        systems = case["engines"] if kind == "batch" else case["fits"]
        ratio = math.log(case["nmax"] / case["nmin"])
        atoms, rows = systems * (case["nmax"] - case["nmin"]) / ratio, 1
        near = min(1.0, systems * 4.0 / 3.0 * math.pi * 12.0 ** 3 * 0.1 / atoms)
    # a step reads the atoms in reach and the tables of its bins; S(Q) adds three matrix-vector products
    bins = 1201 if kind != "chain" else case["rmax"] * 100 + 1
    flops = 50.0 * rows * near * atoms + 40.0 * bins * systems
    if kind == "serve":
        flops += 2.0 * 1201 * 1201 * systems
    return {"bytes": case["steps"] * (20.0 * near * atoms + 16.0 * bins * systems), "flops": case["steps"] * flops}


# ------------------------------------------------------------------- exact
# The path's distances and bins are defined in float32 (fullrmc's own order of
# operations); what is computed from them is evaluated in 64 bits here.
def _wrap(d):
    return d - torch.where(d > 0, torch.floor(d + 0.5), torch.ceil(d - 0.5))


def _dist(a, b, B, pbc):
    """float32 minimum-image distances of broadcast (.., 3) tensors, fullrmc's order."""
    d = [a[..., k] - b[..., k] for k in range(3)]
    if pbc:
        d = [_wrap(x) for x in d]
        d = [(d[0] * B[0][k] + d[1] * B[1][k]) + d[2] * B[2][k] for k in range(3)]
    return torch.sqrt((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2])


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pair_counts(a, rows=None):
    """int64 (2, ne, ne, hs) intra and inter counts: `rows` against all other
    atoms, or (None) every pair i < j."""
    dev = _device()
    c = torch.from_numpy(np.ascontiguousarray(a["boxCoords"])).to(dev)
    el = torch.from_numpy(a["elementIndex"]).to(dev).long()
    mol = torch.from_numpy(a["moleculeIndex"]).to(dev)
    B = [[float(x) for x in r] for r in a["basis"]]
    ne, hs, n = a["numberOfElements"], a["histSize"], c.shape[0]
    lo, up, w = (torch.tensor(float(a[k]), dtype=torch.float32, device=dev)
                 for k in ("minDistance", "maxDistance", "bin"))
    out = torch.zeros(2 * ne * ne * hs, dtype=torch.int64, device=dev)
    idx = torch.arange(n, device=dev) if rows is None else torch.from_numpy(np.asarray(rows)).to(dev).long()
    step = max(1, (1 << 26) // n)
    for i0 in range(0, idx.shape[0], step):
        r = idx[i0:i0 + step]
        first = i0 if rows is None else 0
        d = _dist(c[r][:, None, :], c[None, first:, :], B, a["isPBC"])
        j = torch.arange(first, n, device=dev)
        take = (d >= lo) & (d < up) & ((j[None, :] > r[:, None]) if rows is None else (j[None, :] != r[:, None]))
        k, m = torch.nonzero(take, as_tuple=True)
        b = ((d[k, m] - lo) / w).long()
        i, m = r[k], m + first
        flat = ((torch.where(mol[i] == mol[m], 0, 1) * ne + el[i]) * ne + el[m]) * hs + b
        out += torch.bincount(flat[flat < out.shape[0]], minlength=out.shape[0])
    return out.view(2, ne, ne, hs).cpu().numpy()


def _exact_contacts(case, a):
    dev = _device()
    c = torch.from_numpy(a["boxCoords"]).to(dev)
    el, mol = torch.from_numpy(a["elementIndex"]).to(dev).long(), torch.from_numpy(a["moleculeIndex"]).to(dev)
    lo, up = (torch.from_numpy(a[k].reshape(3, 3)).to(dev) for k in ("lowerLimit", "upperLimit"))
    B, n = [[float(x) for x in r] for r in a["basis"]], c.shape[0]
    every = "indexes" not in a
    idx = torch.arange(n, device=dev) if every else torch.from_numpy(a["indexes"]).to(dev).long()
    num = torch.zeros(18, dtype=torch.int64, device=dev)
    tot = torch.zeros(18, dtype=torch.float64, device=dev)
    for i0 in range(0, idx.shape[0], 1024):
        r = idx[i0:i0 + 1024]
        d = _dist(c[r][:, None, :], c[None], B, True)
        l, h = (t[el[None, :], el[r][:, None]] for t in (lo, up))
        j = torch.arange(n, device=dev)[None, :]
        take = (d >= l) & (d < h) & ((j > r[:, None]) if every else (j != r[:, None]))
        take &= mol[r][:, None] != mol[None, :]
        k, m = torch.nonzero(take, as_tuple=True)
        x, l, h = d[k, m].double(), l[k, m].double(), h[k, m].double()
        if case["reduce"] == "upper":
            x = (h - x).abs()
        elif case["reduce"] == "nearest":
            x = torch.where(x > (l + h) / 2, (h - x).abs(), (l - x).abs())
        at = 9 + el[r[k]] * 3 + el[m]
        num += torch.bincount(at, minlength=18)
        tot.index_add_(0, at, x)
    num, tot = num.cpu().numpy().reshape(2, 3, 3, 1), tot.cpu().numpy().reshape(2, 3, 3, 1)
    return num[0].astype(np.int32), tot[0], num[1].astype(np.int32), tot[1]


def _exact_coordination(a):
    dev = _device()
    c = torch.from_numpy(a["boxCoords"]).to(dev)
    B, n = [[float(x) for x in r] for r in a["basis"]], c.shape[0]
    rows = torch.arange(n, device=dev) if "indexes" not in a else torch.from_numpy(a["indexes"]).to(dev).long()
    inside = torch.zeros(n, dtype=torch.bool, device=dev)
    inside[rows] = True
    out = np.zeros(len(_DEFINITIONS))
    for d in range(len(_DEFINITIONS)):
        lo, up = float(a["lowerShells"][d]), float(a["upperShells"][d])
        core, shell = (torch.from_numpy(a[k][d]).to(dev).long() for k in ("coresIndexes", "shellsIndexes"))
        for mine, other in ((core, shell), (shell, core)):
            mine = mine[inside[mine]]
            for i0 in range(0, mine.shape[0], 1024):
                x = _dist(c[mine[i0:i0 + 1024]][:, None, :], c[other][None], B, True)
                out[d] += int(((x >= lo) & (x <= up)).sum())
    return out


def _exact_sine(way, a):
    if way == "sq_to_Gr":
        y, x, f = (np.asarray(a[k], np.float64) for k in ("qValues", "rValues", "sq"))
        return 2.0 / np.pi * (np.sin(np.outer(x, y)) @ ((y[1] - y[0]) * y * (f - 1.0)))
    y, x = (np.asarray(a[k], np.float64) for k in ("distances", "qrange"))
    if way == "Gr_to_sq":
        w, mul = (y[1] - y[0]) * np.asarray(a["Gr"], np.float64), 1.0
    else:
        w, mul = (y[1] - y[0]) * y * (np.asarray(a["gr"], np.float64) - 1.0), 4.0 * np.pi * float(F32(a["rho"]))
    return 1.0 + mul * (np.sin(np.outer(x, y)) @ w) / x


def _exact_shape(a):
    dr = F32(a["dr"])
    edges = np.arange(F32(a["rmin"]), F32(F32(a["rmax"]) + dr), dr).astype(F32)
    r = ((edges[:-1] + edges[1:]) / F32(2.0)).astype(F32).astype(np.float64)
    Q = np.arange(F32(a["qmin"]), F32(a["qmax"]), F32(a["dq"])).astype(F32).astype(np.float64)
    n = np.asarray(a["elementsCount"], np.float64)
    k = _pair_counts(dict(a, numberOfElements=len(n), histSize=len(r), minDistance=edges[0], maxDistance=edges[-1],
                          bin=dr)).sum(axis=0).astype(np.float64)
    b = n / n.sum() * np.asarray(a["weights"], np.float64)
    g = np.zeros(len(r))
    for i in range(len(n)):
        for j in range(i, len(n)):
            pairs = n[i] * (n[i] - 1) / 2 if i == j else n[i] * n[j]
            weight = (1.0 if i == j else 2.0) * b[i] * b[j] / b.sum() ** 2
            g += weight * a["volume"] / pairs * (k[i, i] if i == j else k[i, j] + k[j, i])
    e = edges.astype(np.float64)
    g /= 4.0 / 3.0 * np.pi * (e[1:] ** 3 - e[:-1] ** 3)
    G = 4.0 * np.pi * r * (n.sum() / a["volume"]) * (g - 1.0)
    S = 1.0 + np.sin(np.outer(Q, r)) @ ((r[1] - r[0]) * G) / Q
    x = np.asarray(a["rValues"], np.float64)
    return 2.0 / np.pi * (np.sin(np.outer(x, Q)) @ ((Q[1] - Q[0]) * Q * (S - 1.0))), G, S


class _Replay:
    """One engine's chain on the host: float32 moves and distances, chi2 in 64 bits from the counts."""

    def __init__(self, s):
        self.s, m = s, s.model
        self.box, self.real = s.box_coords.copy(), s.real_coords.copy()
        self.a = _hist_args(s)
        k = _pair_counts(dict(self.a, boxCoords=self.box)).sum(axis=0)
        self.ne, self.hs = k.shape[0], k.shape[2]
        self.counts = (k + k.transpose(1, 0, 2)) // (1 + np.eye(self.ne, dtype=np.int64))[:, :, None]
        n = np.asarray(m.elements_count, np.float64)
        self.coef = np.zeros((self.ne, self.ne))
        for i in range(self.ne):
            for j in range(i, self.ne):
                pairs = n[i] * (n[i] - 1) / 2 if i == j else n[i] * n[j]
                if pairs > 0:
                    self.coef[i, j] = m.weights[i][j] * m.volume / pairs
        self.rho = n.sum() / m.volume
        e = m.edges.astype(np.float64)
        self.vol = 4.0 / 3.0 * np.pi * (e[1:] ** 3 - e[:-1] ** 3)
        self.r = m.r.astype(np.float64)
        self.M = None
        if s.sq is not None:
            e = (float(m.minDistance) + float(m.bin) * np.arange(self.hs + 1)).astype(F32)
            self.qr = ((e[:-1] + e[1:]) / F32(2.0)).astype(F32).astype(np.float64)
            e = e.astype(np.float64)
            self.qvol = 4.0 / 3.0 * np.pi * (e[1:] ** 3 - e[:-1] ** 3)
            q = s.sq.q.astype(np.float64)
            self.M = torch.from_numpy((self.qr[1] - self.qr[0]) * np.sin(np.outer(self.qr, q)) / q).to(_device())
            self.S = torch.from_numpy(np.asarray(s.sq.S_exp, np.float64)).to(_device())
        self.chi2 = self.error(self.counts)

    def error(self, counts):
        g = np.einsum("ij,ijb->b", self.coef, counts.astype(np.float64))
        d = np.asarray(self.s.model.G_exp, np.float64) - 4 * np.pi * self.r * self.rho * (g / self.vol - 1.0)
        out = float(d @ d)
        if self.M is not None:
            G = torch.from_numpy(4 * np.pi * self.qr * self.rho * (g / self.qvol - 1.0)).to(self.M.device)
            d = self.S - (G @ self.M + 1.0)
            out += float(d @ d)
        return out

    def pairs(self, box, atoms):
        """Counts (pairs of elements, either order) of the atoms with all others, their own pairs once."""
        m, B = self.a, self.a["basis"]
        out = np.zeros(self.ne * self.ne * self.hs, np.int64)
        member = np.zeros(box.shape[0], bool)
        for a in atoms:
            member[a] = True
            d = box[a] - box
            d -= np.trunc(d + np.copysign(F32(0.5), d))
            x = [(d[:, 0] * B[0, k] + d[:, 1] * B[1, k]) + d[:, 2] * B[2, k] for k in range(3)]
            d = np.sqrt((x[0] * x[0] + x[1] * x[1]) + x[2] * x[2])
            at = np.flatnonzero((d >= m["minDistance"]) & (d < m["maxDistance"]) & ~member)
            b = ((d[at] - m["minDistance"]) / m["bin"]).astype(np.int64)
            e = self.s.el[at].astype(np.int64)
            out += np.bincount((self.s.el[a] * self.ne + e) * self.hs + b, minlength=out.shape[0])[:out.shape[0]]
        out = out.reshape(self.ne, self.ne, self.hs)
        return (out + out.transpose(1, 0, 2)) // (1 + np.eye(self.ne, dtype=np.int64))[:, :, None]

    def step(self, atoms, new_real, u):
        M = self.s.rbasis
        new_box = np.stack([(new_real[:, 0] * M[0, k] + new_real[:, 1] * M[1, k]) + new_real[:, 2] * M[2, k]
                            for k in range(3)], axis=1)
        before = self.pairs(self.box, atoms)
        old = self.box[atoms]
        self.box[atoms] = new_box
        counts = self.counts - before + self.pairs(self.box, atoms)
        chi2 = self.error(counts)
        take = not (chi2 > self.chi2 and u > self.s.tolerance)
        if take:
            self.counts, self.chi2 = counts, chi2
            self.real[atoms] = new_real
        else:
            self.box[atoms] = old
        return chi2, take


def _moved_group(real, kind, p):
    """Group translation, or rotation about the centroid, in the engines' float32 order."""
    if kind == 0:
        return real + p[:3]
    c = real[0].copy()
    for k in range(1, real.shape[0]):
        c = c + real[k]
    c = c / F32(real.shape[0])
    R, d = p.reshape(3, 3), real - c
    return np.stack([((d[:, 0] * R[0, k] + d[:, 1] * R[1, k]) + d[:, 2] * R[2, k]) + c[k] for k in range(3)], axis=1)


def _exact_engines(case, seed):
    systems = _engine_systems(case, seed)
    moves = _streams(case, systems, seed)
    c2 = np.empty((case["steps"], len(systems)))
    acc = np.empty((case["steps"], len(systems)), np.int32)
    for e, s in enumerate(systems):
        chain, m = _Replay(s), moves[e]
        for k in range(case["steps"]):
            if s.group_size > 1:
                atoms, new = m[0][k], _moved_group(chain.real[m[0][k]], m[1][k], m[2][k])
            else:
                atoms = m[0][k:k + 1]
                new = chain.real[atoms] + m[1][k]
            c2[k, e], acc[k, e] = chain.step(atoms, new.astype(F32), m[-1][k])
    if case["kind"] == "chain":
        first = moves[0][0][:case["steps"]]
        return c2[:, 0], acc[:, 0], first[:, 0] if first.ndim == 2 else first
    return (c2, acc) if case["kind"] == "batch" else (np.ascontiguousarray(c2.T), np.ascontiguousarray(acc.T))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "chain", "serve"):
        return _exact_engines(case, seed)
    _, a = prepare(case, seed)
    if kind in ("move", "full"):
        k = _pair_counts(a, a.get("indexes")).astype(np.float64)
        return k[0], k[1]
    if kind == "contacts":
        return _exact_contacts(case, a)
    if kind == "coordination":
        return _exact_coordination(a)
    if kind == "distances":
        c = np.asarray(a["coords"], np.float64)
        d = c[a["indexes"]][None, :, :] - c[:, None, :]
        d = (d - np.round(d)) @ np.asarray(a["basis"], np.float64)
        return np.sqrt((d * d).sum(axis=2))
    if kind == "sine":
        return _exact_sine(*a)
    return _exact_shape(a)
