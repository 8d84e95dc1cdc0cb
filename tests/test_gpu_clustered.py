"""Graphs most of whose wedges close: the look-ups go to the table at once and no first step is run twice, by
the bytes that a sample reads; and every way of a graph gives the oracle's samples."""
import numpy as np
import pytest

import zgraph as Z

pytestmark = pytest.mark.gpu


def lattice(n, k, rewired, seed=1):
    """A ring lattice, k neighbours on either side, with a part of its edges sent to random places."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), k)
    j = (i + np.tile(np.arange(1, k + 1), n)) % n
    r = rng.random(len(i)) < rewired
    j[r] = rng.integers(0, n, r.sum())
    e = np.unique(np.sort(np.stack([i, j], 1)[i != j], 1), axis=0)
    e = e[rng.permutation(len(e))]
    flip = rng.random(len(e)) < 0.5
    e[flip] = e[flip][:, ::-1]
    return e.astype(np.uint32), n


def cliques(count, k):
    i, j = np.triu_indices(k, 1)
    at = np.arange(count)[:, None] * k
    e = np.stack([(at + i).ravel(), (at + j).ravel()], 1)
    return e[np.random.default_rng(k).permutation(len(e))].astype(np.uint32), count * k


@pytest.mark.parametrize("make", [lambda: cliques(100, 100), lambda: lattice(20000, 10, 0.0)])
def test_samples_read_no_more_than_one_pass(make):
    """A triangle sample's sectors on packed records, at most: the record and its ends' offsets (which the
    counting build reads though this step does not use them), the drawn entry, two buckets, and the record
    that confirms."""
    e, nv = make()
    g = Z.Graph.from_edges(e, nv)
    assert g.meta().record_layout == Z.RECORDS_PACKED
    assert Z.Program(Z.PROG_TRIANGLE).touch_bytes_per_sample(g, 1 << 21, 5) <= 7 * 32


@pytest.mark.parametrize("layout", [Z.RECORDS_AUTO, Z.RECORDS_COMPACT, Z.RECORDS_WIDE])
@pytest.mark.parametrize("rewired", [0.0, 0.15, 0.5, 1.0])
def test_every_way_gives_the_oracles_samples(rewired, layout):
    import oracle as O
    e, nv = lattice(3000, 6, rewired)
    Z.set_record_layout(layout)
    try:
        g = Z.Graph.from_edges(e, nv)
    finally:
        Z.set_record_layout(Z.RECORDS_AUTO)
    og = O.OracleGraph(e, nv)
    b = Z.Batch(g, max_queries=4)
    n = (1 << 20) + 777  # several rounds of a grid, and a last one that is not full
    for kind in (Z.PROG_TRIANGLE, Z.PROG_FOUR_CLIQUE, Z.PROG_FOUR_CLIQUE_UNBIASED):
        want = O.run(og, O.OracleProgram(kind), n, 7)
        (batch, _), = b.run([{"kind": kind, "n": n, "seed": 7}])
        for got in (Z.Program(kind).run(g, n, 7), batch):
            assert (got.hits, got.fails, got.exact_sum()) == (want.hits, want.fails, want.exact_sum())
