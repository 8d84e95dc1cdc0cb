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
