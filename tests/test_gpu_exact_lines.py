"""Exact counts of houses and 4-edge paths on either side of the lines between their kernels: the most
vertices of the one-launch form (12 272, and 12 288, where its counters alone fill 48 KB), the most edges
of it (20 480) and the most vertices whose wedge counters fit a block (24 576)."""
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
