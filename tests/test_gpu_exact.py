"""zg_exact_count against closed forms on complete graphs, whose out-degrees under the degree
orientation run through every value below n: each class of vertex (one warp, one block, one block
with its tables in global memory) and the edges between the classes are met."""
from math import comb

import numpy as np
import pytest

import zgraph as Z

pytestmark = pytest.mark.gpu


def complete(n, seed=1):
    i, j = np.triu_indices(n, 1)
    e = np.stack([i, j], 1).astype(np.uint32)
    rng = np.random.default_rng(seed)
    return e[rng.permutation(len(e))]


@pytest.mark.parametrize("n", [2, 3, 5, 33, 34, 65, 257, 258, 290, 1025, 1030, 1100])
def test_complete_graph_triangles_and_4_cliques(n):
    e = complete(n)
    w = np.where(e.max(1) < n // 2, 60, 40).astype(np.uint32)  # data >= 50: the complete graph on n // 2
    g = Z.Graph.from_edges(e, n, weights=w)
    assert g.exact_count(Z.EXACT_TRIANGLE) == comb(n, 3)
    assert g.exact_count(Z.EXACT_FOUR_CLIQUE) == comb(n, 4)
    assert g.exact_count_weighted(Z.EXACT_WEIGHTED_TRIANGLE, 50) == comb(n // 2, 3)
    below = g.exact_count_weighted(Z.EXACT_AT_LEAST_ONE_TRIANGLE, 50)
    assert below == sum(comb(n // 2, k) * comb(n - n // 2, 3 - k) for k in (2, 3))


def grid_and_hubs(scale, hubs, seed):
    """A sparse random graph with a few hubs joined to many of its vertices: every class of wedge count."""
    rng = np.random.default_rng(seed)
    nv = 1 << scale
    e = [rng.integers(0, nv, (2 * nv, 2))]
    for h in range(hubs):
        e.append(np.stack([np.full(nv // (4 + h), h), rng.integers(hubs, nv, nv // (4 + h))], 1))
    e = np.concatenate(e)
    e = e[e[:, 0] != e[:, 1]]
    e = np.unique(np.sort(e, 1), axis=0).astype(np.uint32)
    return e[rng.permutation(len(e))], nv


@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 34, 90, 300])
def test_complete_graph_houses_and_paths(n):
    g = Z.Graph.from_edges(complete(n), n)
    # 5 vertices and an order of them, over the pattern's symmetries (2 each)
    assert g.exact_count(Z.EXACT_FIVE_HOUSE) == comb(n, 5) * 60
    assert g.exact_count(Z.EXACT_FIVE_CHAIN) == comb(n, 5) * 60


@pytest.mark.parametrize("scale,hubs", [(8, 2), (12, 6), (14, 3), (15, 3)])
def test_houses_and_paths_match_the_oracle(scale, hubs):
    """Vertex counts on both sides of the one whose wedge counters fit a block."""
    import oracle as O
    e, nv = grid_and_hubs(scale, hubs, 5)
    g, og = Z.Graph.from_edges(e, nv), O.OracleGraph(e, nv)
    for kind in (Z.EXACT_FIVE_HOUSE, Z.EXACT_FIVE_CHAIN):
        assert g.exact_count(kind) == og.exact_fast(kind)
    # the same edges spread over more vertex ids than any block has counters for
    wide = Z.Graph.from_edges((e.astype(np.uint64) * 37).astype(np.uint32), nv * 37)
    for kind in (Z.EXACT_FIVE_HOUSE, Z.EXACT_FIVE_CHAIN):
        assert wide.exact_count(kind) == g.exact_count(kind)
