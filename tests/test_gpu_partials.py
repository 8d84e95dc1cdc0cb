"""Where partial sums change hands: batches whose queries end inside, at and past a chunk (which
shrinks to 2^8 samples for short batches), and runs whose block count takes one or two levels of
reduction.  Counts and exact sums equal those of the same samples in other pieces."""
import pytest

import zgraph as Z

pytestmark = pytest.mark.gpu

STAR = (5, [(0, 1), (0, 2), (0, 3), (0, 4)])


def same(a, b):
    assert (a.samples, a.hits, a.fails, a.overflow) == (b.samples, b.hits, b.fails, b.overflow)
    assert a.exact_sum() == b.exact_sum() and a.estimate == b.estimate
    assert a.sum_w2 == pytest.approx(b.sum_w2, rel=1e-12)


@pytest.fixture(scope="module")
def graphs():
    Z.init(0)
    out = {}
    for name, layout in (("packed", Z.RECORDS_AUTO), ("wide", Z.RECORDS_WIDE)):
        Z.set_record_layout(layout)
        try:
            out[name] = Z.Graph.gen_rmat(12, 8, seed=3)
        finally:
            Z.set_record_layout(Z.RECORDS_AUTO)
    return out


@pytest.mark.parametrize("sizes", [(1,), (255, 256, 257), (8192,) * 6, (4095, 4096, 4097, 70001), (3000001, 5, 2000003)])
def test_batch_equals_runs(graphs, sizes):
    g = graphs["packed"]
    b = Z.Batch(g, max_queries=8)
    tri, star = Z.Program(Z.PROG_TRIANGLE), Z.Program(Z.PROG_PATTERN, pattern=STAR)
    qs, progs = [], []
    for i, n in enumerate(sizes):
        progs.append(star if i % 2 else tri)
        qs.append({"kind": progs[-1].kind, "n": n, "seed": 7 + i, "stream_id": i, "first_sample": 1000 * i})
        if i % 2:
            qs[-1]["program"] = star
    for _ in range(2):  # the second submit reuses the buffers
        for q, p, (c, rest) in zip(qs, progs, b.run(qs)):
            same(c, p.run(g, q["n"], q["seed"], stream_id=q["stream_id"], first_sample=q["first_sample"]))
            assert (rest.samples, rest.hits, rest.sum_w2) == (0, 0, 0.0)
    h2d, d2h = b.copy_bytes()
    assert h2d > 0 and d2h == 2 * 112 * len(sizes)


@pytest.mark.parametrize("name,n", [("packed", 1), ("packed", 10007), ("packed", 1 << 20), ("wide", 256 * 2048),
                                    ("wide", 256 * 2048 + 1), ("wide", 256 * 2305), ("wide", 1 << 22)])
def test_run_equals_its_pieces(graphs, name, n):
    g, p = graphs[name], Z.Program(Z.PROG_FOUR_CHAIN)
    whole = p.run(g, n, 5, first_sample=11)
    cut = max(1, n // 3)
    parts = [p.run(g, min(cut, n - at), 5, first_sample=11 + at) for at in range(0, n, cut)]
    merged = Z.merge_counters(parts)
    assert (whole.samples, whole.hits, whole.fails) == (n, merged.hits, merged.fails)
    assert whole.exact_sum() == merged.exact_sum()
    assert whole.sum_w2 == pytest.approx(merged.sum_w2, rel=1e-12)
