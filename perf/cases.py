"""The calls whose speed is tracked, as a user's program makes them through the Python interface.

Each case is a dict of plain values.  `prepare` makes what the program holds before the call (edge
lists, device graphs, programs, batches, the network), `run` is one pass through the public entry
points, `work` is what that pass cannot do without, and `exact` restates the estimators in plain
torch where the outputs are floating point numbers.

Graph sizes are the repository's own configurations (R-MAT scale 13 ef 12, scale 20 ef 3, the
edge-factor-24 R-MAT family, the 42 M-edge Chung-Lu graph) or lie between them.  Launch shapes are the
library's defaults: nothing is tuned first.
"""
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "sampling-graph-mining_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import zgraph as Z  # noqa: E402

PROGRAMS = {"triangle": (Z.PROG_TRIANGLE, 0, None), "four_clique": (Z.PROG_FOUR_CLIQUE, 0, None),
            "four_clique_unbiased": (Z.PROG_FOUR_CLIQUE_UNBIASED, 0, None),
            "three_chain": (Z.PROG_THREE_CHAIN, 0, None), "four_chain": (Z.PROG_FOUR_CHAIN, 0, None),
            "chain5": (Z.PROG_CHAIN, 5, None),
            "five_star": (Z.PROG_PATTERN, 0, (5, [(0, 1), (0, 2), (0, 3), (0, 4)])),
            "five_house": (Z.PROG_PATTERN, 0, (5, [(0, 1), (0, 2), (1, 2), (1, 3), (2, 4), (3, 4)]))}
# the reads one sample cannot do without (32-byte sectors) and its draws
SECTORS = {"triangle": 3, "four_clique": 3, "four_clique_unbiased": 3, "three_chain": 1, "four_chain": 4,
           "chain5": 6, "five_star": 8, "five_house": 9, "three_motif": 3}
DRAWS = {"triangle": 2, "four_clique": 2, "four_clique_unbiased": 2, "three_chain": 2, "four_chain": 4,
         "chain5": 4, "five_star": 4, "five_house": 6, "three_motif": 2}
EXACT = {"triangle": Z.EXACT_TRIANGLE, "wedge": Z.EXACT_WEDGE, "three_path": Z.EXACT_THREE_PATH,
         "five_star": Z.EXACT_FIVE_STAR, "four_clique": Z.EXACT_FOUR_CLIQUE, "five_house": Z.EXACT_FIVE_HOUSE,
         "five_chain": Z.EXACT_FIVE_CHAIN, "weighted_triangle": Z.EXACT_WEIGHTED_TRIANGLE,
         "at_least_one_triangle": Z.EXACT_AT_LEAST_ONE_TRIANGLE}
PHILOX_OPS = 80  # ten rounds of two wide products and four xors; one block serves two draws
FOUR = "triangle,four_clique,three_chain,four_chain"


def listed():
    return [
        # calculate() on a small graph: the shortest call there is; its launches and the host path count
        {"name": "calc_small", "op": "run", "gen": "rmat", "scale": 13, "ef": 12, "programs": "triangle", "n": 10007},
        # the four applications' estimators on a graph about the size of the L2
        {"name": "run_near_l2", "op": "run", "gen": "rmat", "scale": 20, "ef": 3, "programs": FOUR, "n": 1 << 24},
        # the same on a graph read from HBM (the batched configuration's base graph)
        {"name": "run_hbm", "op": "run", "gen": "chung_lu", "nv": 4800000, "degree": 18.0, "programs": FOUR,
         "n": 1 << 25},
        # a few short queries at once: the batch path's fixed cost
        {"name": "batch_small", "op": "batch", "gen": "rmat", "scale": 13, "ef": 12, "programs": FOUR, "n": 1 << 13,
         "queries": 6, "predicates": 0},
        # mixed queries, uneven budgets, some on filtered graphs (triangles, 3-motifs, predicates)
        {"name": "batch_mixed", "op": "batch", "gen": "chung_lu", "nv": 1000000, "degree": 18.0,
         "programs": "triangle,three_motif", "n": 1 << 22, "queries": 48, "predicates": 4},
        # the largest: the headline's estimators in one batch on a graph of tens of GB
        {"name": "batch_large", "op": "batch", "gen": "rmat_device", "scale": 25, "ef": 24,
         "programs": "four_clique,five_star,five_house", "n": 1 << 27, "queries": 3, "predicates": 0},
        # an application's start: the edge list from the host, shuffled, built, first estimate
        {"name": "load_run", "op": "load", "gen": "rmat", "scale": 20, "ef": 3, "programs": "triangle", "n": 1 << 20},
        # AllPredicate: filter by edge data, shuffle, rebuild, estimate
        {"name": "filter_run", "op": "filter", "gen": "rmat", "scale": 20, "ef": 3, "programs": "triangle",
         "n": 1 << 20, "threshold": 50},
        # the reference's error-latency profile (plain sizing) of a 1 % / 95 % query
        {"name": "size_plain", "op": "elp", "gen": "rmat", "scale": 20, "ef": 3, "programs": "triangle", "n": 1 << 23},
        # a 1 % / 95 % answer with the learned sizing
        {"name": "query_learned", "op": "query", "gen": "rmat", "scale": 20, "ef": 3, "programs": "triangle",
         "n": 1 << 25, "error": 0.01},
        # exact counts that answers are checked against: triangles and 4-cliques
        {"name": "exact_cliques", "op": "exact", "gen": "rmat", "scale": 20, "ef": 3, "kinds": "triangle,four_clique"},
        # exact houses and 4-edge paths, at the largest size the repository counts them
        {"name": "exact_house_chain", "op": "exact", "gen": "rmat", "scale": 13, "ef": 12,
         "kinds": "five_house,five_chain"},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(["run", "run", "batch", "batch", "load", "filter", "elp", "query", "exact", "exact"])
    c = {"op": op}
    if op in ("run", "batch") and rng.random() < 0.4:
        c.update(gen="chung_lu", nv=_log_int(rng, 20000, 4800000), degree=round(rng.uniform(8.0, 24.0), 1))
    else:
        c.update(gen="rmat", scale=rng.randint(11, 20), ef=rng.randint(3, 12))
    if op == "run":
        c["programs"] = rng.choice([FOUR, "triangle", "four_clique", "three_chain", "four_chain", "chain5", "five_star",
                                    "five_house", "four_clique_unbiased"])
        c["n"] = _log_int(rng, 1 << 12, 1 << 25)
    elif op == "batch":
        c["programs"] = rng.choice([FOUR, "triangle,three_motif", "four_clique,five_star,five_house"])
        c["n"] = _log_int(rng, 1 << 13, 1 << 23)
        c["queries"] = rng.randint(3, 48)
        c["predicates"] = rng.choice([0, 0, 2, 4])
    elif op in ("load", "filter"):
        c["programs"] = rng.choice(["triangle", "four_clique", "three_chain", "four_chain"])
        c["n"] = _log_int(rng, 1 << 14, 1 << 22)
        if op == "filter":
            c["threshold"] = rng.randint(10, 90)
    elif op == "elp":
        c["programs"] = rng.choice(["triangle", "three_chain", "four_chain", "four_clique"])
        c["n"] = 1 << 23
    elif op == "query":
        c["programs"] = rng.choice(["triangle", "three_chain", "four_chain", "five_star"])
        c["n"] = 1 << 25
        c["error"] = rng.choice([0.01, 0.02, 0.05])
    else:
        c["kinds"] = rng.choice(["triangle,four_clique", "triangle,four_clique", "wedge,five_star,three_path",
                                 "weighted_triangle,at_least_one_triangle", "five_house,five_chain"])
        if c["kinds"] == "five_house,five_chain":  # they grow with the squares of the degrees
            c.update(scale=rng.randint(8, 13), ef=rng.randint(3, 12))
    return c


# ---- inputs -------------------------------------------------------------------------------------
def _rmat_edges(scale, ef, seed):
    """An undirected simplified R-MAT edge list in random order and orientation: (m, 2) int64 on the GPU.
    Drawn twice over and cut, so that m is the same for every seed."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = 2 * ef << scale
    u = torch.zeros(n, dtype=torch.int64, device="cuda")
    v = torch.zeros_like(u)
    for _ in range(scale):
        r = torch.rand(n, generator=gen, device="cuda")
        u = u * 2 + (r >= 0.76)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    key = (torch.minimum(u, v) << 32) | torch.maximum(u, v)
    key = torch.unique(key[u != v])
    key = key[torch.randperm(key.numel(), generator=gen, device="cuda")][:(ef << scale) * 98 // 100]
    lo, hi = key >> 32, key & 0xFFFFFFFF
    flip = torch.rand(key.numel(), generator=gen, device="cuda") < 0.5
    return torch.stack([torch.where(flip, hi, lo), torch.where(flip, lo, hi)], 1)


def _host_edges(e):
    return e.to(torch.int32).cpu().numpy().view(np.uint32)


def _weights(m, seed):
    """Edge data in [0, 100), every value equally often."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    w = torch.randperm(m, generator=gen, device="cuda") % 100
    return w.to(torch.int32).cpu().numpy().view(np.uint32)


def _is_weighted(c):
    return c["op"] == "filter" or c.get("predicates", 0) > 0 or "weighted" in c.get("kinds", "")


def _graph(c, seed):
    w = _is_weighted(c)
    if c["gen"] == "rmat":
        e = _host_edges(_rmat_edges(c["scale"], c["ef"], seed))
        return Z.Graph.from_edges(e, 1 << c["scale"], weights=_weights(len(e), seed) if w else None)
    if c["gen"] == "rmat_device":
        return Z.Graph.gen_rmat(c["scale"], c["ef"], seed=seed, sampling_only=True)
    return Z.Graph.gen_chung_lu(c["nv"], 2.3, c["degree"], seed=seed, max_weight=100 if w else 0, weight_seed=7,
                                sampling_only=True)


def _program(name):
    kind, param, pattern = PROGRAMS[name]
    return Z.Program(kind, param, pattern)


def _queries(c, seed):
    """Budgets spread over a factor of 64 below n (equal ones where there is one query a program)."""
    rng = np.random.default_rng(seed)
    names = c["programs"].split(",")
    progs = {k: _program(k) for k in names if k != "three_motif"}
    qs = []
    for i in range(c["queries"]):
        name = names[i % len(names)]
        n = c["n"] if c["queries"] <= len(names) else max(1, int(c["n"] * 2.0 ** -rng.uniform(0, 6)))
        q = {"kind": Z.QUERY_THREE_MOTIF if name == "three_motif" else PROGRAMS[name][0], "n": n,
             "seed": int(rng.integers(1, 1 << 40)), "stream_id": 2 * i}
        if name in progs:
            q["param"] = PROGRAMS[name][1]
            if PROGRAMS[name][2]:
                q["program"] = progs[name]
        if c["predicates"] and i % 2:
            j = i // 2 % c["predicates"]
            q.update(pred_op=Z.PRED_LT if j % 2 else Z.PRED_GE, t0=20 + 60 * j // c["predicates"])
        qs.append(q)
    return qs, progs


def prepare(case, seed):
    Z.init(0)
    c = dict(case)
    s = {"case": c, "seed": seed}
    if c["op"] == "load":
        s["edges"] = _host_edges(_rmat_edges(c["scale"], c["ef"], seed))
    else:
        s["graph"] = _graph(c, seed)
    if c["op"] == "batch":
        s["queries"], s["programs"] = _queries(c, seed)
        s["batch"] = Z.Batch(s["graph"], max_queries=64, cache_bytes=8 << 30, filter_seed=seed)
    elif c["op"] != "exact":
        s["programs"] = [_program(k) for k in c["programs"].split(",")]
    if c["op"] == "query":
        s["net"] = Z.Mlp.load(os.path.join(_PKG, "elp_mlp.npz"))
    return s


# ---- one pass -----------------------------------------------------------------------------------
def _counters(k):
    return {"samples": int(k.samples), "hits": int(k.hits), "fails": int(k.fails),
            "sum_num": np.array(k.sum_num[:], np.uint64).view(np.int64), "den_log2": int(k.den_log2),
            "estimate": float(k.estimate), "sum_w": float(k.sum_w), "sum_w2": float(k.sum_w2), "sum_w4": float(k.sum_w4)}


def run(state):
    c, seed, op = state["case"], state["seed"], state["case"]["op"]
    if op == "run":
        return [_counters(p.run(state["graph"], c["n"], seed, stream_id=i)) for i, p in enumerate(state["programs"])]
    if op == "batch":
        out = state["batch"].run(state["queries"])
        fields = [(k, t) if q["kind"] == Z.QUERY_THREE_MOTIF else (k,) for q, (k, t) in zip(state["queries"], out)]
        rows = [x for r in fields for x in r]
        return {"samples": np.array([k.samples for k in rows], np.int64),
                "hits": np.array([k.hits for k in rows], np.int64),
                "fails": np.array([k.fails for k in rows], np.int64),
                "sum_num": np.array([k.sum_num[:] for k in rows], np.uint64).view(np.int64),
                "estimate": np.array([k.estimate for k in rows]), "sum_w": np.array([k.sum_w for k in rows]),
                "sum_w2": np.array([k.sum_w2 for k in rows]), "sum_w4": np.array([k.sum_w4 for k in rows])}
    if op == "load":
        g = Z.Graph.from_edges(state["edges"], 1 << c["scale"], shuffle_seed=seed)
        k = _counters(state["programs"][0].run(g, c["n"], seed))
        out = {"counters": k, "parent": g.parent_index.view(np.int64), "max_degree": int(g.max_degree)}
        g.free()
        return out
    if op == "filter":
        f = state["graph"].filter(Z.PRED_GE, c["threshold"], shuffle_seed=seed)
        k = _counters(state["programs"][0].run(f, c["n"], seed))
        out = {"counters": k, "parent": f.parent_index.view(np.int64), "max_degree": int(f.max_degree)}
        f.free()
        return out
    if op == "elp":
        r, groups = Z.elp_plain(state["graph"], state["programs"][0], 0.01, 0.95, seed, want_groups=True)
        return {"groups": groups, "n_required": float(r.n_required_f), "K": float(r.K),
                "estimate_sampled": float(r.estimate_sampled), "big_estimate": float(r.big_estimate),
                "sampled_edges": int(r.sampled_edges), "sampled_max_degree": int(r.sampled_max_degree)}
    if op == "query":
        r, n = Z.learned_query(state["net"], state["graph"], state["programs"][0], c["error"], 0.95, seed, seed + 100,
                               stream_id=0x51, max_samples=1 << 28)
        return {"budget": n, "samples": int(r.samples), "hits": int(r.hits), "met": int(r.bound_met),
                "estimate": float(r.estimate), "half_width": float(r.half_width)}
    out = []
    for k in c["kinds"].split(","):
        kind = EXACT[k]
        v = (state["graph"].exact_count_weighted(kind, 50) if "weighted" in c["kinds"]
             else state["graph"].exact_count(kind))
        out.append(np.array([v & 0xFFFFFFFF, v >> 32 & 0xFFFFFFFF, v >> 64], np.int64))
    return out


# ---- what a pass cannot do without --------------------------------------------------------------
def work(case):
    c = case
    if c["gen"] == "chung_lu":
        m, nv = int(c["degree"] * c["nv"] / 2), c["nv"]
    else:
        m, nv = c["ef"] << c["scale"], 1 << c["scale"]
    graph = 42 * m + 4 * nv  # records, adjacency and edge table as sampled
    if c["op"] == "exact":
        # every edge once, and per edge the shorter of two neighbour lists (about the mean degree)
        deep = "five_house" in c["kinds"]
        return {"bytes": 8 * m, "flops": len(c["kinds"].split(",")) * m * (2 * m / nv) ** (2 if deep else 1)}
    names = c["programs"].split(",")
    if c["op"] == "batch":
        each = c["n"] if c["queries"] <= len(names) else c["n"] / 4
        n = [(names[i % len(names)], each) for i in range(c["queries"])]
    else:
        n = [(k, c["n"]) for k in names]
    bytes_ = min(graph, sum(32 * SECTORS[k] * x for k, x in n))
    flops = sum(PHILOX_OPS * DRAWS[k] / 2 * x for k, x in n)
    if c["op"] == "load":
        bytes_ += 8 * m + 8 * m + graph  # the list in, the permutation out, the graph's arrays written
    elif c["op"] == "filter":
        kept = m * (100 - c["threshold"]) / 100
        bytes_ += 12 * m + kept / m * (8 * m + graph)
    elif c["op"] == "elp":
        bytes_ += 8 * m + 0.1 * graph
    return {"bytes": bytes_, "flops": flops}


# ---- the estimators in plain torch --------------------------------------------------------------
_M32 = 0xFFFFFFFF


def _word(seed, stream, n, d):
    """The 64-bit word of draw d of samples 0 .. n-1 as (high, low) 32-bit halves: Philox4x32-10, counter
    (sample, d // 2, stream), key seed; an even draw takes output words 1:0, an odd one 3:2."""
    i = torch.arange(n, dtype=torch.int64, device="cuda")
    c0, c1 = i & _M32, i >> 32
    c2, c3 = torch.full_like(i, d >> 1), torch.full_like(i, stream)
    k0, k1 = seed & _M32, seed >> 32 & _M32
    for _ in range(10):
        p0, p1 = 0xD2511F53 * c0, 0xCD9E8D57 * c2
        c0, c1, c2, c3 = (p1 >> 32 & _M32) ^ c1 ^ k0, p1 & _M32, (p0 >> 32 & _M32) ^ c3 ^ k1, p0 & _M32
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return (c3, c2) if d & 1 else (c1, c0)


def _below(word, size):
    """The word mapped to [0, size) by multiply-high (size below 2^32)."""
    hi, lo = word
    return (hi * size + (lo * size >> 32 & _M32)) >> 32 & _M32


class _Lists:
    """Every vertex's neighbours in edge-id order, and the edge ids by pair."""

    def __init__(self, e, nv):
        m = e.shape[0]
        self.e, self.m = e, m
        ids = torch.arange(m, dtype=torch.int64, device="cuda")
        at = torch.cat([e[:, 0], e[:, 1]]) << 32 | torch.cat([ids, ids])
        self.at, order = torch.sort(at)
        self.nbr = torch.cat([e[:, 1], e[:, 0]])[order]
        self.off = torch.searchsorted(self.at, torch.arange(nv + 1, dtype=torch.int64, device="cuda") << 32)
        key = torch.minimum(e[:, 0], e[:, 1]) << 32 | torch.maximum(e[:, 0], e[:, 1])
        self.pair, self.pair_id = torch.sort(key)

    def from_id(self, v, eid):
        """The first place in v's list with edge id >= eid, and the list's end."""
        return torch.searchsorted(self.at, v << 32 | eid), self.off[v + 1]

    def entry(self, p):
        p = p.clamp(0, 2 * self.m - 1)
        return self.nbr[p], self.at[p] & _M32

    def closed(self, x, y, eid):
        key = torch.minimum(x, y) << 32 | torch.maximum(x, y)
        p = torch.searchsorted(self.pair, key).clamp(max=self.m - 1)
        return (self.pair[p] == key) & (self.pair_id[p] >= eid)

    def step(self, word, anchors, eid):
        """One conditional step over the anchors' entries from eid on: the number of entries, the chosen
        anchor's index and the chosen entry."""
        ranges = [self.from_id(v, eid) for v in anchors]
        size = sum(hi - lo for lo, hi in ranges)
        r = _below(word, size)
        slot, place = torch.full_like(r, len(anchors) - 1), torch.zeros_like(r)
        open_ = torch.ones_like(r, dtype=torch.bool)
        for k, (lo, hi) in enumerate(ranges):
            here = open_ & (r < hi - lo)
            slot, place = torch.where(here, k, slot), torch.where(here, lo + r, place)
            r, open_ = torch.where(open_ & ~here, r - (hi - lo), r), open_ & ~here
        nbr, got = self.entry(place)
        return size, slot, nbr, got


def _estimate(name, g, n, seed, stream):
    """(weights, hits) of the estimator on samples 0 .. n-1: weight 1/p where it hit, else 0."""
    def word(d):
        return _word(seed, stream, n, d)
    first = 1 if name == "four_chain" else 0
    e0 = _below(word(first), torch.full((n,), g.m, dtype=torch.int64, device="cuda"))
    a, b = g.e[e0, 0], g.e[e0, 1]
    w = torch.full((n,), float(g.m), dtype=torch.float64, device="cuda")
    if name == "four_chain":
        pick = 1 + _below(word(0), torch.full((n,), 3, dtype=torch.int64, device="cuda"))
        s, slot, c, e1 = g.step(word(2), [a, b], e0 + 1)
        far = c
        s2, _, d, e2 = g.step(word(3), [far], torch.where(pick == 1, e1, e0) + 1)
        hit = (s > 0) & (s2 > 0) & (d != a) & (d != b) & ((pick == 1) | (e2 < e1))
        t, _, x, _ = g.step(word(2), [a], e0 + 1)
        t2, _, y, _ = g.step(word(3), [b], e0 + 1)
        split = (t > 0) & (t2 > 0) & (x != y) & (x != b) & (y != a)
        hit = torch.where(pick == 3, split, hit)
        w = w * 3 * torch.where(pick == 3, t, s) * torch.where(pick == 3, t2, s2)
        return torch.where(hit, w, 0.0), hit
    s, slot, c, e1 = g.step(word(1), [a, b], e0 + 1)
    w, ok = w * s, s > 0
    if name == "three_chain":
        return torch.where(ok, w, 0.0), ok
    other = torch.where(slot == 0, b, a)
    if name == "triangle":
        hit = ok & g.closed(other, c, e1 + 1)
        return torch.where(hit, w, 0.0), hit
    s2, slot2, d, e2 = g.step(word(2), [a, b, c], e1 + 1)
    w = w * s2
    hit = ok & (s2 > 0) & (d != a) & (d != b) & (d != c) & g.closed(other, c, e2 + 1)
    for k, v in enumerate((a, b, c)):
        hit &= (slot2 == k) | g.closed(v, d, e2 + 1)
    return torch.where(hit, w, 0.0), hit


def _exact_counters(name, g, n, seed, stream):
    keys = ("samples", "hits", "fails", "sum_num", "den_log2")
    w, _ = _estimate(name, g, n, seed, stream)
    return {**{k: None for k in keys}, "estimate": float(w.sum() / n), "sum_w": float(w.sum()),
            "sum_w2": float((w ** 2).sum()), "sum_w4": float((w ** 4).sum())}


def exact(case, seed):
    c = case
    if c["op"] != "run" or c["gen"] != "rmat" or not set(c["programs"].split(",")) <= set(FOUR.split(",")):
        return None
    g = _Lists(_rmat_edges(c["scale"], c["ef"], seed), 1 << c["scale"])
    return [_exact_counters(k, g, c["n"], seed, i) for i, k in enumerate(c["programs"].split(","))]
