"""The device graph build against numpy: the seeded edge order (Philox keys, ties by position) around
the sizes where its buckets double, and every exported array in each record layout."""
import numpy as np
import pytest

import zgraph as Z

pytestmark = pytest.mark.gpu

M32 = np.uint64(0xFFFFFFFF)


def shuffle_keys(m, seed, stream=0xFFFFFFF0):
    """Philox4x32-10 words 1:0 at counter (i, 0, stream), key seed."""
    i = np.arange(m, dtype=np.uint64)
    c = [i & M32, i >> np.uint64(32), np.zeros(m, np.uint64), np.full(m, stream, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & M32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & M32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return (c[1] << np.uint64(32)) | c[0]


def simple_edges(m, seed):
    rng = np.random.default_rng(seed)
    nv = max(4, int(2 * m ** 0.6))
    e = np.unique(np.sort(rng.integers(0, nv, (3 * m + 20, 2)), 1), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    e = e[rng.permutation(len(e))][:m]
    flip = rng.random(len(e)) < 0.5
    e[flip] = e[flip][:, ::-1]
    return e.astype(np.uint32), nv + 3


@pytest.mark.parametrize("m,layout", [(1, Z.RECORDS_AUTO), (2, Z.RECORDS_WIDE), (31, Z.RECORDS_COMPACT),
                                      (2047, Z.RECORDS_AUTO), (2048, Z.RECORDS_WIDE), (2049, Z.RECORDS_COMPACT),
                                      (4096, Z.RECORDS_PACKED), (4097, Z.RECORDS_AUTO), (100003, Z.RECORDS_AUTO),
                                      (300001, Z.RECORDS_WIDE)])
def test_build_matches_numpy(m, layout):
    e, nv = simple_edges(m, m)
    m = len(e)
    seed = 0x1234567890 + m
    Z.set_record_layout(layout)
    try:
        g = Z.Graph.from_edges(e, nv, weights=np.arange(m, dtype=np.uint32), shuffle_seed=seed)
    finally:
        Z.set_record_layout(Z.RECORDS_AUTO)
    perm = np.argsort(shuffle_keys(m, seed), kind="stable")
    assert np.array_equal(g.parent_index, perm.astype(np.uint64))
    e = e[perm]
    d = g.download()
    assert np.array_equal(d["edges"], e) and np.array_equal(d["weights"], perm.astype(np.uint32))
    ids = np.arange(m, dtype=np.uint32)
    v, n, i = (np.concatenate(x) for x in ((e[:, 0], e[:, 1]), (e[:, 1], e[:, 0]), (ids, ids)))
    off = np.concatenate([[0], np.cumsum(np.bincount(v, minlength=nv))])
    assert np.array_equal(d["offsets"], off) and g.max_degree == np.diff(off).max()
    o = np.lexsort((i, v))
    assert np.array_equal(d["adj_e"], np.stack([n[o], i[o]], 1))
    place = np.empty(2 * m, np.int64)
    place[o] = np.arange(2 * m)
    assert np.array_equal(d["suffix"], np.stack([off[e[:, k] + 1] - 1 - place[k * m:(k + 1) * m] for k in (0, 1)], 1))
    o = np.lexsort((n, v))
    assert np.array_equal(d["adj_n"], np.stack([n[o], i[o]], 1))
    f = g.filter(Z.PRED_LT, m // 2, shuffle_seed=7)
    kept = np.flatnonzero(d["weights"] < m // 2)
    assert np.array_equal(f.parent_index, kept[np.argsort(shuffle_keys(len(kept), 7), kind="stable")])


@pytest.mark.parametrize("edges", [[(0, 1), (2, 2)], [(0, 1), (5, 1)], [(0, 1), (1, 0)], [(0, 1), (0, 1), (2, 3)]])
def test_invalid_edges_are_refused(edges):
    with pytest.raises(Z.ZgError) as err:
        Z.Graph.from_edges(np.array(edges, np.uint32), 4)
    assert err.value.code == Z.ZG_ERR_INVALID_GRAPH


@pytest.mark.parametrize("m", [1, 3, 4, 5, 31, 32, 33, 5000])
def test_every_edge_is_found_and_no_other(m):
    """The filter and the table behind it, at the sizes where the filter gains a word."""
    e, nv = simple_edges(m, 7 * m)
    g = Z.Graph.from_edges(e, nv)
    rng = np.random.default_rng(m)
    pairs = [tuple(int(x) for x in p) for p in np.concatenate([e, e[:, ::-1], rng.integers(0, nv, (2000, 2))])]
    ids = {(int(a), int(b)): i for i, (a, b) in enumerate(e)}
    ids.update({(b, a): i for (a, b), i in list(ids.items())})
    got = Z.conditional_close(g, [(0, [a, b], [(a, b)]) for a, b in pairs])
    for p, (closed, found, at) in zip(pairs, got):
        assert closed == (p in ids) and at == ([ids[p]] if closed else [])
