"""Reads of one handle on different streams, issued one after the other by one
thread without waiting for the device: each still has the answer that it has
alone.  Part of a read's device scratch is the handle's and is in use until
the read has finished, so the next one waits for it on the device."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import _dev
from test_gpu_read_balance import _u32

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph(engine, oracle):
    V = 1 << 14
    e = oracle.rmat_edges(3, 14, 32)
    g = engine.Lpma(V)
    g.update(ins=_dev(e))
    yield g, V, e
    g.close()


def _fill(g, srcs, wins, bufs, stream):
    """The call that writes the lists; returns before they are written."""
    offs, nbrs, vals = bufs
    total = ctypes.c_size_t()
    rc = g._L.lpma_query_neighbors(g._h, srcs.data_ptr(), wins.data_ptr(), srcs.numel(), offs.data_ptr(),
                                   nbrs.data_ptr(), vals.data_ptr(), nbrs.numel(), ctypes.byref(total), stream.cuda_stream)
    assert rc == 0
    return total.value


@pytest.mark.parametrize("n", [512, 9000])  # one CTA weighs the queries, many do
def test_neighbour_lists_on_two_streams(graph, n):
    import torch
    g, V, e = graph
    rng = np.random.default_rng(n)
    qs = [rng.integers(0, V, n), np.arange(V, dtype=np.int64), rng.integers(0, 64, 200)]
    srcs = [_u32(q) for q in qs]
    wins = [torch.full((q.size,), 0xFFFFFFFF, dtype=torch.int64, device="cuda") for q in qs]
    want = [g.query_neighbors(s, w) for s, w in zip(srcs, wins)]
    bufs = [tuple(torch.zeros_like(x) for x in w) for w in want]
    streams = [torch.cuda.Stream() for _ in qs]
    torch.cuda.synchronize()
    for turn in range(30):
        for b in bufs:
            for x in b:
                x.zero_()
        torch.cuda.synchronize()
        for i in np.random.default_rng(turn).permutation(3):
            assert _fill(g, srcs[i], wins[i], bufs[i], streams[i]) == want[i][1].numel()
        torch.cuda.synchronize()
        for w, b in zip(want, bufs):
            for x, y in zip(w, b):
                assert torch.equal(x, y)


def test_view_beside_pagerank(graph, oracle):
    import torch
    g, V, e = graph
    rank = oracle.pagerank(g.export_sorted()[0], V, 0.85, 10)
    ref = oracle.OracleLpma(V)
    ref.update(ins=e)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    out = torch.zeros(V, dtype=torch.float64, device="cuda")
    for turn in range(20):
        extra = np.array([(turn << 42) | (turn << 20)], np.uint64)  # a self loop, in and out: the view is made anew
        g.update(ins=_dev(extra))
        g.update(dels=_dev(extra))
        torch.cuda.synchronize()
        out.zero_()
        torch.cuda.synchronize()
        assert g._L.lpma_pagerank(g._h, 0.85, 10, out.data_ptr(), s1.cuda_stream) == 0
        g.stream = s2
        try:
            ro, ci, va = g.to_csr()
        finally:
            g.stream = None
        torch.cuda.synchronize()
        for x, y in zip((ro, ci, va), ref.csr()):
            assert np.array_equal(x, y)
        assert np.allclose(out.cpu().numpy(), rank, rtol=1e-10, atol=0)
