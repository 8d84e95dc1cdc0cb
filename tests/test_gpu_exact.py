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
