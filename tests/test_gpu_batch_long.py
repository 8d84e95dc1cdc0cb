"""Batches long enough for chunks of many samples a thread, on every record layout, against single runs on
wide records (which take their samples one by one): the counters and exact sums are equal.  And the plain
sizing's regression where it shares its work among threads."""
import numpy as np
import pytest

import zgraph as Z

pytestmark = pytest.mark.gpu

KINDS = (Z.PROG_TRIANGLE, Z.PROG_FOUR_CLIQUE, Z.PROG_FOUR_CLIQUE_UNBIASED, Z.QUERY_THREE_MOTIF, Z.PROG_FOUR_CHAIN)


def build(layout):
    Z.set_record_layout(layout)
    try:
        return Z.Graph.gen_rmat(12, 8, seed=3)
    finally:
        Z.set_record_layout(Z.RECORDS_AUTO)


def singles(g, qs):
    for q in qs:
        if q["kind"] == Z.QUERY_THREE_MOTIF:
            yield Z.run_three_motif(g, q["n"], q["n"], q["seed"], 0, 1)
        else:
            yield Z.Program(q["kind"]).run(g, q["n"], q["seed"]), None


@pytest.mark.parametrize("n", [1 << 20, 2500003, 12000007])
def test_long_batches_equal_single_runs(n):
    qs = [{"kind": k, "n": n + i, "seed": 3 + i} for i, k in enumerate(KINDS)]
    want = list(singles(build(Z.RECORDS_WIDE), qs))
    for layout in (Z.RECORDS_PACKED, Z.RECORDS_COMPACT, Z.RECORDS_WIDE):
        g = build(layout)
        assert g.meta().record_layout == layout
        for got, ref in zip(Z.Batch(g, max_queries=8).run(qs), want):
            for a, b in zip(got, ref):
                if b is not None:
                    assert (a.samples, a.hits, a.fails, a.overflow) == (b.samples, b.hits, b.fails, b.overflow)
                    assert a.exact_sum() == b.exact_sum() and a.estimate == b.estimate
                    assert a.sum_w2 == pytest.approx(b.sum_w2, rel=1e-12)


@pytest.mark.parametrize("n_groups", [4095, 4096, 4097, 5003, 1 << 14])
def test_plain_sizing_shared_among_threads(n_groups):
    import oracle as O
    groups = np.random.default_rng(n_groups).gamma(2.0, 1e6, n_groups)
    groups[::7] = 0.0
    args = (groups, 16, float(groups.mean()), 1 << 23, 1.0, 2.0, 10 ** 6, 900, 10 ** 7, 4000, 0.05, 0.95)
    got = Z.elp_solve(*args)
    want = O.elp_solve(*args)
    assert abs(got.n_required_f - want) <= 1e-9 * abs(want)
    assert all(Z.elp_solve(*args).n_required_f == got.n_required_f for _ in range(5))
