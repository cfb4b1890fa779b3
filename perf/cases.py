"""The workloads whose speed is followed: what users of this framework have it
do, through its public entry points, over the range of sizes in real use.

A case is a dict of plain values; `listed` names the followed ones, `draw`
gives more of the same ranges.  Sizes and edges are those of the tests, of
bench.py's workloads and of the reference's example, kdbench and tests, or
smaller and odd ones of the same kinds.  Inputs are seeded and synthetic.
"""
import math

import numpy as np
import torch

from corruscant_b200 import _native, clustering
from corruscant_b200.twopoint import angular, threedim


def listed():
    return [
        # one pair_count call of a small script or of a per-edge loop written
        # against the reference's C entry point: a small tree, a few raw query
        # points, one radius; launches, allocations and waits are all it costs
        {"name": "pair_count_1k", "kind": "pair_count", "n_tree": 4000, "n_query": 1000,
         "fields": 1, "rmax": 0.1},
        # the reference's own C benchmark: 400k uniform points, 4 fields,
        # queried with themselves at one radius, as raw points
        {"name": "pair_count_400k", "kind": "pair_count", "n_tree": 400000, "n_query": 400000,
         "fields": 4, "rmax": 0.05},
        # the reference's example: 4k data, 80k randoms, 6 edges, no fields
        {"name": "autocorr_example", "kind": "autocorr", "n_data": 4000, "n_rand": 80000,
         "fields": 1, "rmin": 10 ** -2.5, "rmax": 0.1, "edges": 6, "mode": 0},
        # a galaxy survey with jackknife fields at full size: 1M clustered
        # data, 20M randoms, 21 edges, 64 fields
        {"name": "autocorr_20m", "kind": "autocorr", "n_data": 1000000, "n_rand": 20000000,
         "fields": 64, "rmin": 1e-3, "rmax": 0.1, "edges": 21, "mode": 0},
        # the same kind of survey with every distance in FP64 (the caller's
        # choice of mode), odd sizes
        {"name": "autocorr_fp64", "kind": "autocorr", "n_data": 150001, "n_rand": 2000003,
         "fields": 27, "rmin": 1e-3, "rmax": 0.1, "edges": 21, "mode": 1},
        # w(theta) on a patch of sky with 100 jackknife fields, 16 edges
        {"name": "angular_5m", "kind": "angular", "n_data": 500000, "n_rand": 5000000,
         "fields": 100, "rmin": 1e-3, "rmax": 2.0, "edges": 16},
        # cross-correlation of two catalogs of different sizes, each with its
        # own randoms: four counts, odd sizes
        {"name": "crosscorr", "kind": "crosscorr", "n_data": 30011, "n_data2": 50021,
         "n_rand": 300007, "n_rand2": 500009, "fields": 8, "rmin": 2e-3, "rmax": 0.1,
         "edges": 13},
        # many mock catalogs of ragged sizes against shared randoms, one batch
        {"name": "mocks", "kind": "mocks", "catalogs": 24, "n_min": 20000, "n_max": 500000,
         "n_rand": 1000000, "fields": 16, "rmin": 2e-3, "rmax": 0.1, "edges": 13},
        # gridded positions (simulation cells, rounded catalogs): duplicates,
        # ties and many pairs exactly on an edge; both cross counts
        {"name": "lattice", "kind": "lattice", "n_data": 1000003, "n_rand": 1000003,
         "fields": 27, "edges": 30},
        # a tree alone through the Python class, node array read: small
        {"name": "tree_80k", "kind": "tree", "n": 80000, "fields": 1},
        # a tree alone through the C entry point with its node array: large
        {"name": "tree_5m", "kind": "construct", "n": 5000011, "fields": 64},
        # a whole script from arrays on the host: both trees, then the counts
        {"name": "survey_1m", "kind": "survey", "n_data": 100003, "n_rand": 1000003,
         "fields": 16, "rmin": 1e-3, "rmax": 0.1, "edges": 16, "mode": 0},
    ]


def _size(rng, lo, hi):
    """A size spread over its logarithm, odd more often than not."""
    n = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    return n | 1 if rng.random() < 0.7 else n


def draw(rng):
    kind = rng.choice(["pair_count", "autocorr", "autocorr", "angular", "crosscorr", "mocks",
                       "lattice", "tree", "construct", "survey"])
    few = rng.choice([1, 4, 8])
    bins = {"rmin": rng.choice([1e-3, 2e-3, 10 ** -2.5]), "rmax": rng.choice([0.05, 0.08, 0.1]),
            "edges": rng.randint(4, 22)}
    if kind == "pair_count":
        return {"kind": kind, "n_tree": _size(rng, 1000, 1000000),
                "n_query": _size(rng, 100, 400000), "fields": few,
                "rmax": rng.choice([0.01, 0.05, 0.1])}
    if kind == "autocorr":
        nd = _size(rng, 1000, 400000)
        return {"kind": kind, "n_data": nd, "n_rand": nd * rng.choice([5, 10, 20]) + rng.randint(0, 9),
                "fields": few if nd < 20000 else rng.choice([1, 8, 27, 64]),
                "mode": int(rng.random() < 0.25), **bins}
    if kind == "angular":
        nd = _size(rng, 10000, 500000)
        return {"kind": kind, "n_data": nd, "n_rand": 10 * nd + rng.randint(0, 9),
                "fields": rng.choice([1, 4, 25, 100]), "rmin": 1e-3,
                "rmax": rng.choice([0.5, 1.0, 2.0]), "edges": rng.randint(6, 18)}
    if kind == "crosscorr":
        nd, nd2 = _size(rng, 2000, 100000), _size(rng, 2000, 100000)
        return {"kind": kind, "n_data": nd, "n_data2": nd2, "n_rand": 10 * nd + 7,
                "n_rand2": 10 * nd2 + 3, "fields": few, **bins}
    if kind == "mocks":
        return {"kind": kind, "catalogs": rng.randint(4, 24), "n_min": 20000,
                "n_max": _size(rng, 40000, 400000), "n_rand": _size(rng, 200000, 1000000),
                "fields": 16, **bins}
    if kind == "lattice":
        n = _size(rng, 20000, 1000000)
        return {"kind": kind, "n_data": n, "n_rand": n + rng.randint(0, 1000), "fields": 27,
                "edges": rng.randint(8, 30)}
    if kind == "survey":
        nd = _size(rng, 4000, 200000)
        return {"kind": kind, "n_data": nd, "n_rand": 10 * nd + rng.randint(0, 9), "fields": few,
                "mode": 0, **bins}
    if kind == "tree":
        return {"kind": kind, "n": _size(rng, 1000, 1000000), "fields": few}
    return {"kind": kind, "n": _size(rng, 100000, 5000000), "fields": rng.choice([1, 16, 64])}


# ------------------------------------------------------------------ inputs

class _Source:
    """Seeded random numbers, made on the GPU where that is quicker."""

    def __init__(self, seed):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.gen = torch.Generator(device=self.dev)
        self.gen.manual_seed(int(seed) * 2654435761 % (1 << 62))

    def uniform(self, *shape):
        return torch.rand(shape, generator=self.gen, device=self.dev, dtype=torch.float64)

    def normal(self, *shape):
        return torch.randn(shape, generator=self.gen, device=self.dev, dtype=torch.float64)

    def below(self, m, *shape):
        return torch.randint(0, m, shape, generator=self.gen, device=self.dev)


def _host(points, fields):
    f = None if fields is None else fields.to(torch.int32).cpu().numpy()
    return np.ascontiguousarray(points.cpu().numpy()), f


def _grid_fields(p, nf):
    """Jackknife fields: the cells of a regular grid over the unit cube."""
    if nf == 1:
        return None
    nx, ny, nz = {4: (4, 1, 1), 8: (2, 2, 2), 16: (4, 4, 1), 27: (3, 3, 3), 64: (4, 4, 4)}[nf]
    c = [(p[:, i] * m).floor().clamp(0, m - 1).to(torch.int64) for i, m in enumerate((nx, ny, nz))]
    return (c[0] * ny + c[1]) * nz + c[2]


def _cube(src, n, nf):
    p = src.uniform(n, 3)
    return _host(p, _grid_fields(p, nf))


def _clustered(src, n, nf):
    """Neyman-Scott: children around uniform parents, wrapped periodically."""
    parents = src.uniform(max(n // 100, 20 * nf), 3)
    p = (parents[src.below(parents.shape[0], n)] + 0.005 * src.normal(n, 3)) % 1.0
    return _host(p, _grid_fields(p, nf))


def _sky(src, n, nf, blobs):
    """(RA, DEC) on RA 0-90, DEC -10..60, uniform on the sphere; a share of the
    points in blobs of 0.05 degrees; fields: cells equal in RA and sin DEC."""
    s0, s1 = math.sin(math.radians(-10.0)), math.sin(math.radians(60.0))
    nb = int(n * blobs)
    ra, s = 90.0 * src.uniform(n), s0 + (s1 - s0) * src.uniform(n)
    if nb:
        at = src.below(max(1, nb // 50), nb)
        ra[:nb], s[:nb] = ra[at], s[at]
        ra[:nb] = (ra[:nb] + 0.05 * src.normal(nb)).clamp(0.0, 90.0)
        s[:nb] = (s[:nb] + math.radians(0.05) * src.normal(nb)).clamp(s0, s1)
    f = None
    if nf > 1:
        m = int(round(math.sqrt(nf)))
        f = ((ra / 90.0 * m).floor().clamp(0, m - 1) * m +
             ((s - s0) / (s1 - s0) * m).floor().clamp(0, m - 1)).to(torch.int64)
    dec = torch.rad2deg(torch.arcsin(s))
    return ra.cpu().numpy(), dec.cpu().numpy(), None if f is None else f.to(torch.int32).cpu().numpy()


def _lattice(src, n, nf, copies):
    p = src.below(1024, n, 3).to(torch.float64) / 1024.0
    if copies:
        rows = torch.nonzero(src.uniform(n) < 0.10).flatten()
        p[rows] = p[src.below(n, rows.numel())]
    return _host(p, _grid_fields(p, nf))


def _lattice_edges(ne):
    k = np.unique(np.round(np.geomspace(1, 10486, ne + 2)).astype(np.int64))
    return np.sqrt(k.astype(np.float64)) / 1024.0


def _radii(case):
    if case["kind"] == "lattice":
        return _lattice_edges(case["edges"])
    return np.logspace(math.log10(case["rmin"]), math.log10(case["rmax"]), case["edges"])


def _catalogs(case, seed):
    """The case's catalogs on the host: name -> (points, fields)."""
    src, kind, nf = _Source(seed), case["kind"], case["fields"]
    if kind == "pair_count":
        tree = _cube(src, case["n_tree"], nf)
        return {"T": tree, "Q": tree if case["n_query"] == case["n_tree"] else
                _cube(src, case["n_query"], nf)}
    if kind in ("autocorr", "survey"):
        return {"D": _clustered(src, case["n_data"], nf), "R": _cube(src, case["n_rand"], nf)}
    if kind == "angular":
        cats = {}
        for name, n, blobs in (("D", case["n_data"], 0.5), ("R", case["n_rand"], 0.0)):
            ra, dec, f = _sky(src, n, nf, blobs)
            cats[name] = (angular.cartesian(ra, dec), f)
        return cats
    if kind == "crosscorr":
        return {"D": _clustered(src, case["n_data"], nf),
                "D2": _clustered(src, case["n_data2"], nf),
                "R": _cube(src, case["n_rand"], nf), "R2": _cube(src, case["n_rand2"], nf)}
    if kind == "mocks":
        m = case["catalogs"]
        step = (case["n_max"] / case["n_min"]) ** (1.0 / max(1, m - 1))
        cats = {"M%02d" % i: _clustered(src, int(case["n_min"] * step ** i), nf) for i in range(m)}
        cats["R"] = _cube(src, case["n_rand"], nf)
        return cats
    if kind == "lattice":
        return {"D": _lattice(src, case["n_data"], nf, True),
                "R": _lattice(src, case["n_rand"], nf, False)}
    return {"D": _clustered(src, case["n"], nf)}


class _Trees:
    """The C entry point's trees of a program, given back with it."""

    def __init__(self):
        self.held = []

    def add(self, t):
        self.held.append(t)
        return t

    def __del__(self):
        while self.held:
            _native.destroy(self.held.pop())


def _nodes(ctree, owner):
    """The node array that the C struct points to, as whole words; the tree
    lives as long as the array is held."""
    words = _native.c_longlong * (5 * ctree.memsize)
    buf = words.from_address(_native.ctypes.addressof(ctree.node_data.contents))
    buf.owner = owner
    return np.frombuffer(buf, dtype=np.int64).reshape(ctree.memsize, 5)


# ---------------------------------------------------------------- one pass

def prepare(case, seed):
    cats = _catalogs(case, seed)
    state = {"case": dict(case), "cats": cats}
    if case["kind"] in ("tree", "construct", "survey"):
        return state  # the pass builds its own trees
    if case["kind"] in ("mocks", "lattice"):
        held = state["made"] = _Trees()
        state["trees"] = {k: held.add(_native.build_tree(p, f, case["fields"]))
                          for k, (p, f) in cats.items()}
    elif case["kind"] == "pair_count":
        state["trees"] = {"T": clustering.tree(*cats["T"])}
    else:
        state["trees"] = {k: clustering.tree(p, f) for k, (p, f) in cats.items()}
    return state


def _jobs(case):
    if case["kind"] == "lattice":
        return [("R", "D"), ("D", "R")]
    names = ["M%02d" % i for i in range(case["catalogs"])]
    return [j for m in names for j in ((m, m), ("R", m))] + [("R", "R")]


def _results(res, nf):
    out = {"counts": list(res.count_arrays), "estimate": res.estimate()}
    if nf > 1:  # the error bars a user of fields is after
        out["covariance"] = res.covariance("jackknife")
    return out


def run(state):
    case, cats, trees = state["case"], state["cats"], state.get("trees")
    kind, nf = case["kind"], case["fields"]
    if kind == "pair_count":
        points, fields = cats["Q"]
        return _native.pair_count(trees["T"].ctree, points, fields, nf, case["rmax"])
    if kind == "autocorr":
        return _results(threedim.autocorr(trees["D"], trees["R"], _radii(case),
                                          mode=case["mode"]), nf)
    if kind == "angular":
        return _results(angular.autocorr(trees["D"], trees["R"], _radii(case)), nf)
    if kind == "crosscorr":
        return _results(threedim.crosscorr(trees["D"], trees["D2"], trees["R"], trees["R2"],
                                           _radii(case)), nf)
    if kind in ("mocks", "lattice"):
        return _native.count_batch([(trees[t], trees[q]) for t, q in _jobs(case)], _radii(case))
    if kind == "survey":
        d, r = clustering.tree(*cats["D"]), clustering.tree(*cats["R"])
        return _results(threedim.autocorr(d, r, _radii(case)), nf)
    points, fields = cats["D"]
    if kind == "tree":
        t = clustering.tree(points, fields)
        return _nodes(t.ctree, t)
    made = _Trees()
    return _nodes(made.add(_native.build_tree(points, fields, nf)), made)


# ------------------------------------------------------------ what it costs

def _memsize(n):
    return 1 << (int(math.log2(n)) + 1)


def _pairs(n1, n2, r, same):
    """Pairs of two catalogs closer than r at uniform density in the unit cube
    (clustered catalogs have more), each unordered pair of one catalog once."""
    return n1 * n2 * min(1.0, 4.0 / 3.0 * math.pi * r ** 3) * (0.5 if same else 1.0)


def work(case):
    """Bytes: points (and fields) read once, results written once.  Flops: 8 for
    every distance of a pair closer than the last edge (3 subtractions, a
    multiply, 2 fused multiply-adds)."""
    kind, nf = case["kind"], case["fields"]
    point = 24 if nf == 1 else 28
    if kind in ("tree", "construct"):
        return {"bytes": case["n"] * point + 40 * _memsize(case["n"]), "flops": 0}
    if kind == "pair_count":
        return {"bytes": (case["n_tree"] + case["n_query"]) * point + 8 * nf * nf,
                "flops": 8 * _pairs(case["n_tree"], case["n_query"], case["rmax"], False)}
    if kind == "mocks":
        m = case["catalogs"]
        step = (case["n_max"] / case["n_min"]) ** (1.0 / max(1, m - 1))
        size = {"M%02d" % i: int(case["n_min"] * step ** i) for i in range(m)}
        size["R"] = case["n_rand"]
        jobs = _jobs(case)
    elif kind == "lattice":
        size = {"D": case["n_data"], "R": case["n_rand"]}
        jobs = _jobs(case)
    elif kind == "crosscorr":
        size = {"D": case["n_data"], "D2": case["n_data2"], "R": case["n_rand"],
                "R2": case["n_rand2"]}
        jobs = [("D", "D2"), ("R2", "D"), ("R", "D2"), ("R", "R2")]
    else:
        size = {"D": case["n_data"], "R": case["n_rand"]}
        jobs = [("D", "D"), ("R", "D"), ("R", "R")]
    if kind == "angular":  # caps of the patch's solid angle
        area = math.radians(90.0) * (math.sin(math.radians(60.0)) - math.sin(math.radians(-10.0)))
        share = 2.0 * math.pi * (1.0 - math.cos(math.radians(case["rmax"]))) / area
        pairs = sum(size[a] * size[b] * share * (0.5 if a == b else 1.0) for a, b in jobs)
    else:
        r = float(_radii(case)[-1])
        pairs = sum(_pairs(size[a], size[b], r, a == b) for a, b in jobs)
    out = 8 * case["edges"] * nf * nf * len(jobs)
    if kind == "survey":
        out += 40 * sum(_memsize(n) for n in size.values())
    return {"bytes": sum(size.values()) * point + out, "flops": 8 * pairs}


# ------------------------------------------------------- the same in 64 bits

def _pairs_under(tree, query, radii, nf):
    """(radii, query field, tree field) counts of the pairs closer than each
    radius, every distance computed."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    (tp, tf), (qp, qf) = ((torch.as_tensor(p, device=dev),
                           torch.zeros(len(p), dtype=torch.int64, device=dev) if f is None else
                           torch.as_tensor(f, device=dev).to(torch.int64))
                          for p, f in (tree, query))
    rsq = torch.as_tensor(np.asarray(radii) ** 2, device=dev)
    ne = len(radii)
    hist = torch.zeros((ne + 1) * nf * nf, dtype=torch.int64, device=dev)
    step = max(1, 40_000_000 // len(tp))
    for a in range(0, len(qp), step):
        q = qp[a:a + step]
        d2 = torch.zeros((len(q), len(tp)), dtype=torch.float64, device=dev)
        for i in range(3):
            d2 += (tp[None, :, i] - q[:, i, None]) ** 2
        bins = torch.bucketize(d2, rsq, right=True)
        bins = (bins * nf + qf[a:a + step, None]) * nf + tf[None, :]
        hist += torch.bincount(bins.flatten(), minlength=hist.numel())
    return torch.cumsum(hist.reshape(ne + 1, nf, nf)[:ne], 0).cpu().numpy()


def exact(case, seed):
    """The counts from all distances in 64 bits, and the estimates from the
    counts, where that is quick; the large cases' and the lattice's values are
    whole numbers decided at the edge, the trees' are bytes."""
    kind, nf = case["kind"], case["fields"]
    if kind not in ("pair_count", "autocorr", "survey", "crosscorr"):
        return None
    if kind == "pair_count":
        cost = case["n_tree"] * case["n_query"]
    elif kind == "crosscorr":
        cost = (case["n_data"] + case["n_rand"]) * (case["n_data2"] + case["n_rand2"])
    else:
        cost = (case["n_data"] + case["n_rand"]) ** 2
    if cost > 4e10:
        return None
    cats = _catalogs(case, seed)
    if kind == "pair_count":
        return _pairs_under(cats["T"], cats["Q"], [case["rmax"]], nf)[0].reshape(-1)
    radii = _radii(case)
    if kind == "crosscorr":
        pairs = [("D", "D2") if case["n_data"] > case["n_data2"] else ("D2", "D"), ("R2", "D"),
                 ("R", "D2"), ("R", "R2") if case["n_rand"] > case["n_rand2"] else ("R2", "R")]
    else:
        pairs = [("D", "D"), ("R", "D"), ("R", "R")]
    counts = [np.diff(_pairs_under(cats[t], cats[q], radii, nf), axis=0) for t, q in pairs]
    sizes = {k: np.bincount(f, minlength=nf) if f is not None else np.array([len(p)])
             for k, (p, f) in cats.items()}
    norm = [("D", "D2"), ("D", "R2"), ("D2", "R"), ("R", "R2")] if kind == "crosscorr" else \
        [("D", "D"), ("D", "R"), ("R", "R")]

    def estimator(totals, norms):
        v = [t / float(n) for t, n in zip(totals, norms)]
        dd, dr, rd, rr = v if len(v) == 4 else (v[0], v[1], v[1], v[2])
        return (dd - dr - rd + rr) / rr

    whole = [c.sum(axis=(1, 2)) for c in counts]
    xi = estimator(whole, [sizes[a].sum() * sizes[b].sum() for a, b in norm])
    out = {"counts": counts, "estimate": xi}
    if nf > 1:
        cov = np.zeros((len(xi), len(xi)))
        for k in range(nf):
            keep = np.arange(nf) != k
            part = [c[:, keep][:, :, keep].sum(axis=(1, 2)) for c in counts]
            d = estimator(part, [sizes[a][keep].sum() * sizes[b][keep].sum() for a, b in norm]) - xi
            d = d * np.sqrt(part[-1] / whole[-1])
            cov += d[:, None] * d[None, :]
        out["covariance"] = cov
    return out
