"""What a build needs on the device at its peak: at most 144 bytes an edge, edge list included, on graphs of
wide records (112 of a graph for sampling only), so that the largest graphs fit."""
import contextlib

import numpy as np
import pytest

import zgraph as Z

pytestmark = pytest.mark.gpu

SLACK = 64 << 20  # the pool grows by whole blocks, and vertices take 24 bytes each


def circulant(nv, k):
    """k edges from every vertex to the next ones, in random order."""
    i = np.arange(nv, dtype=np.uint32)
    e = np.concatenate([np.stack([i, (i + j) % nv], 1) for j in range(1, k + 1)])
    return e[np.random.default_rng(k).permutation(len(e))], nv


@contextlib.contextmanager
def room(nbytes):
    """Wide records, and no more free memory than this."""
    import torch
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    Z.set_record_layout(Z.RECORDS_WIDE)
    held = torch.empty(max(0, free - nbytes), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()
        Z.set_record_layout(Z.RECORDS_AUTO)


@pytest.mark.parametrize("weighted", [False, True])
def test_full_build_fits_144_bytes_an_edge(weighted):
    e, nv = circulant(1 << 20, 24)
    w = np.arange(len(e), dtype=np.uint32) if weighted else None
    Z.Graph.from_edges(e[:1000], nv).free()
    with room((144 + 8 * weighted) * len(e) + SLACK):
        g = Z.Graph.from_edges(e, nv, weights=w)
    assert g.num_local_edges == len(e) and g.max_degree == 48


def test_sampling_build_fits_112_bytes_an_edge():
    """The filtered graph of a batch: its build, its edges before and after their shuffle, with their data
    and places in the base graph."""
    e, nv = circulant(1 << 20, 24)
    g = Z.Graph.from_edges(e, nv, weights=np.arange(len(e), dtype=np.uint32) % 100)
    b = Z.Batch(g, max_queries=1)
    with room((112 + 12) * len(e) + SLACK):
        f = b.filtered_graph(Z.PRED_GE, 0)
    assert f.num_local_edges == len(e) and f.max_degree == 48
