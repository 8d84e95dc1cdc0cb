"""Batches and streams: a submit waits for the batch before it on any stream, the default one included,
and one on a capturing stream is refused before it has touched anything."""
import pytest

import zgraph as Z

pytestmark = pytest.mark.gpu


def same(a, b):
    assert (a.samples, a.hits, a.fails) == (b.samples, b.hits, b.fails)
    assert a.exact_sum() == b.exact_sum() and a.estimate == b.estimate


@pytest.fixture(scope="module")
def graph():
    Z.init(0)
    return Z.Graph.gen_rmat(12, 8, seed=3, max_weight=100)


def queries(count, n, seed):
    kinds = (Z.PROG_TRIANGLE, Z.PROG_THREE_CHAIN, Z.PROG_FOUR_CHAIN)
    return [{"kind": kinds[i % 3], "n": n + i, "seed": seed + i} for i in range(count)]


@pytest.mark.parametrize("stream", ["default", "own"])
@pytest.mark.parametrize("first,second", [(64, 1), (1, 64), (40, 41)])
def test_second_submit_waits_for_the_first(graph, stream, first, second):
    import torch
    s = torch.cuda.Stream().cuda_stream if stream == "own" else None
    b = Z.Batch(graph, max_queries=64)
    qs = queries(second, 3001, 90)
    b.submit(queries(first, 1 << 20, 7), cuda_stream=s)
    b.submit(qs, cuda_stream=s)
    for q, (c, _) in zip(qs, b.wait()):
        same(c, Z.Program(q["kind"]).run(graph, q["n"], q["seed"]))
    b.submit(queries(first, 1 << 20, 7), cuda_stream=s)
    f = b.filtered_graph(Z.PRED_GE, 50)  # may take the place of a graph that the running batch uses
    assert 0 < f.num_local_edges < graph.num_local_edges
    b.submit(qs, cuda_stream=s)
    b.free()  # with the last one running


def test_a_capturing_stream_is_refused_and_its_capture_goes_on(graph):
    import torch
    b = Z.Batch(graph, max_queries=8)
    qs = queries(3, 5000, 11)
    b.submit(qs)
    x = torch.zeros(16, device="cuda")
    torch.cuda.synchronize()
    held, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(held, stream=s, capture_error_mode="thread_local"):
        x.add_(1)
        for more in ({}, {"pred_op": Z.PRED_GE, "t0": 30}):  # the second's filter is not built yet
            with pytest.raises(Z.ZgError) as err:
                b.submit([dict(q, **more) for q in qs[:2]], cuda_stream=s.cuda_stream)
            assert err.value.code == Z.ZG_ERR_CUDA
    held.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 16
    for q, (c, _) in zip(qs, b.wait()):  # the batch before is as it was
        same(c, Z.Program(q["kind"]).run(graph, q["n"], q["seed"]))
