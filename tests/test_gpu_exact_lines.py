"""Exact counts of houses and 4-edge paths on either side of the lines between their kernels: the most
vertices of the one-launch form (12 288, where its counters alone fill 48 KB), the most edges of it
(20 480) and the most vertices whose wedge counters fit a block (24 576)."""
import numpy as np
import pytest

import zgraph as Z

pytestmark = pytest.mark.gpu


def sparse(nv, m, seed):
    """m distinct edges on nv vertices, the last one among them, a few of them hubs."""
    rng = np.random.default_rng(seed)
    e = np.concatenate([rng.integers(0, nv, (2 * m, 2)), np.stack([rng.integers(0, 4, m), rng.integers(4, nv, m)], 1)])
    e = e[e[:, 0] != e[:, 1]]
    e = np.unique(np.sort(e, 1), axis=0)
    e = e[rng.permutation(len(e))][:m]
    e[0] = (0, nv - 1)
    e = np.unique(np.sort(e, 1), axis=0)
    return e[rng.permutation(len(e))].astype(np.uint32)


@pytest.mark.parametrize("nv,m", [(12271, 500), (12272, 20480), (12273, 20480), (12284, 900), (12285, 900), (12288, 20480),
                                  (12288, 20500), (12289, 20480), (700, 20490), (24575, 30000), (24576, 30000),
                                  (24577, 30000)])
def test_houses_and_paths_at_the_lines(nv, m):
    import oracle as O
    e = sparse(nv, m, nv + m)
    g, og = Z.Graph.from_edges(e, nv), O.OracleGraph(e, nv)
    for kind in (Z.EXACT_FIVE_HOUSE, Z.EXACT_FIVE_CHAIN):
        assert g.exact_count(kind) == og.exact_fast(kind)


def stars_and_more(kind):
    """Graphs of hubs: their leaves make most of their degree, and few wedges or none close."""
    rng = np.random.default_rng(5)
    if kind == "star":
        return np.stack([np.full(12000, 7000), np.delete(np.arange(12001), 7000)], 1), 12001
    if kind == "K2,n":
        return np.stack([np.repeat([11, 9990], 9998), np.tile(np.delete(np.arange(10000), [11, 9990]), 2)], 1), 10000
    n = {"small": 9000, "dense": 13000, "wide": 25000}[kind]
    hub = np.stack([np.zeros(n - 1, np.int64), np.arange(1, n)], 1)  # triangles on some of a star's leaves
    return np.concatenate([hub, np.stack([np.arange(1, 2001, 2), np.arange(2, 2002, 2)], 1),
                           np.unique(np.sort(rng.integers(2001, 2200, (900, 2)), 1), axis=0)]), n


@pytest.mark.parametrize("kind", ["star", "K2,n", "small", "dense", "wide"])
def test_houses_and_paths_around_hubs(kind):
    import oracle as O
    e, nv = stars_and_more(kind)
    e = e[e[:, 0] != e[:, 1]]
    e = e[np.random.default_rng(3).permutation(len(e))].astype(np.uint32)
    g, og = Z.Graph.from_edges(e, nv), O.OracleGraph(e, nv)
    for k in (Z.EXACT_FIVE_HOUSE, Z.EXACT_FIVE_CHAIN):
        assert g.exact_count(k) == og.exact_fast(k)


def test_counts_of_several_threads():
    """Counts at once on graphs of different sizes, each on a stream of its own."""
    import threading

    import torch
    graphs = [Z.Graph.from_edges(sparse(nv, 20500, nv), nv) for nv in (12289, 15000, 19000, 24576)]
    want = [[g.exact_count(k) for k in (Z.EXACT_FIVE_HOUSE, Z.EXACT_FIVE_CHAIN)] for g in graphs]
    wrong = []

    def count(g, w, s):
        try:
            for _ in range(200):
                got = [g.exact_count(k, stream=s.cuda_stream) for k in (Z.EXACT_FIVE_HOUSE, Z.EXACT_FIVE_CHAIN)]
                if got != w:
                    wrong.append(got)
        except Z.ZgError as err:
            wrong.append(str(err))

    threads = [threading.Thread(target=count, args=(g, w, torch.cuda.Stream())) for g, w in zip(graphs, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == []
