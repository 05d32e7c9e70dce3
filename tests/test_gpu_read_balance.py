"""Read paths whose work is split by segments, at the edges of the split:
hubs whose slots fill a few segments more or less than one range of the BFS
frontier (4 segments of 32 slots), vertices without edges, every source the
same; neighbour lists of one query, of many, at the size up to which one CTA
places them, and of so many that a hub's rounds are capped; PageRank over
bins of 1,024 destinations and chunks of 16,384 edges."""
import numpy as np
import pytest

from test_gpu_parity import _dev

pytestmark = pytest.mark.gpu


def _u32(a):
    import torch
    return torch.from_numpy(np.asarray(a, np.uint32).view(np.int32)).cuda()


def _hub_graph(engine, deg, V=3000):
    """Vertex 5 points at `deg` vertices, vertex v < 40 at v + 1, the last
    neighbour of the hub at V - 1."""
    rng = np.random.default_rng(deg)
    nbr = np.sort(rng.permutation(np.arange(50, V - 1))[:deg]).astype(np.uint64)
    keys = [(np.uint64(5) << np.uint64(42)) | (nbr << np.uint64(20))]
    v = np.arange(40, dtype=np.uint64)
    keys.append((v << np.uint64(42)) | ((v + np.uint64(1)) << np.uint64(20)))
    if deg:
        keys.append(np.array([(int(nbr[-1]) << 42) | ((V - 1) << 20)], np.uint64))
    keys = np.unique(np.concatenate(keys))
    g = engine.Lpma(V)
    g.update(ins=_dev(keys))
    return g, g.export_sorted()


@pytest.mark.parametrize("deg", [0, 1, 31, 32, 33, 60, 127, 128, 129, 500, 2900])
def test_bfs_hub_ranges(engine, oracle, deg):
    g, (k, _) = _hub_graph(engine, deg)
    for sources, depth in (([5], 0), ([5], 1), ([5, 5, 2999], 2), ([0], 0), ([0], 3), ([0], 4), ([0], 5), ([0], 9),
                           ([2999], 0), ([3000, 4000], 0)):
        dist, levels, reached = g.bfs(_u32(sources), depth)
        srcs = [s for s in sources if s < 3000]
        want = oracle.bfs(k, 3000, srcs, depth) if srcs else np.full(3000, 2**31 - 1)
        assert np.array_equal(dist.cpu().numpy().astype(np.int64), want), (deg, sources, depth)
        seen = want[want != 2**31 - 1]
        assert reached == seen.size
        # a level counts when it had a frontier to expand
        most = int(seen.max()) + 1 if seen.size else 0
        assert levels == (min(most, depth) if depth else most), (deg, sources, depth, levels)
    g.close()


def _lists(k, v, srcs, wins, V):
    """(offsets, neighbours, values), vectorised over the queries."""
    src, dst = (k >> np.uint64(42)).astype(np.int64), (k >> np.uint64(20)) & np.uint64(0x3FFFFF)
    t = (k & np.uint64(0xFFFFF)).astype(np.int64)
    edge = dst != 0x3FFFFE
    src, dst, t, v = src[edge], dst[edge], t[edge], v[edge]
    start = np.searchsorted(src, np.arange(V + 1))
    s = np.asarray(srcs, np.int64)
    inside = s < V
    a, b = np.where(inside, start[np.minimum(s, V - 1)], 0), np.where(inside, start[np.minimum(s, V - 1) + 1], 0)
    row = np.repeat(np.arange(s.size), b - a)
    at = np.arange(row.size) - np.repeat(np.cumsum(b - a) - (b - a), b - a) + np.repeat(a, b - a)
    w = np.asarray(wins, np.uint64)
    lb, ub = (w >> np.uint64(32)).astype(np.int64), (w & np.uint64(0xFFFFFFFF)).astype(np.int64)
    ok = (t[at] >= lb[row]) & (t[at] <= ub[row])
    offs = np.concatenate([[0], np.cumsum(np.bincount(row[ok], minlength=s.size))])
    return offs, dst[at][ok].astype(np.int64), v[at][ok]


def _check_lists(g, k, v, srcs, wins, V):
    offs, nb, nv = g.query_neighbors(_u32(srcs), _dev(wins))
    eo, en, ev = _lists(k, v, srcs, wins, V)
    assert np.array_equal(offs.cpu().numpy().view(np.uint32).astype(np.int64), eo)
    assert np.array_equal(nb.cpu().numpy().astype(np.int64), en)
    assert np.array_equal(nv.cpu().numpy(), ev)


@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1025, 4864, 8191, 8192, 8193, 30000])
def test_neighbor_lists_of_n_queries(engine, n):
    g, (k, v) = _hub_graph(engine, 2900)
    rng = np.random.default_rng(n)
    srcs = rng.integers(0, 3100, n)  # some beyond the last vertex
    srcs[rng.random(n) < 0.02] = 5   # the hub, again and again
    srcs[0] = 5
    wins = np.full(n, 0xFFFFF, np.uint64)
    wins[rng.random(n) < 0.2] = np.uint64(3 << 32 | 9)  # holds nothing
    _check_lists(g, k, v, srcs, wins, 3000)
    _check_lists(g, k, v, np.full(n, 2999), wins, 3000)  # empty lists only
    g.close()


def test_neighbor_lists_with_capped_rounds(engine):
    """2^20 queries: a query counts as at most 2,047 rounds of 4 segments;
    the hub's 400,000 neighbours take more."""
    V, n = 1 << 19, 1 << 20
    rng = np.random.default_rng(1)
    t = np.zeros(400000, np.uint64)
    t[::1000] = 7
    keys = (np.uint64(11) << np.uint64(42)) | (rng.permutation(V - 20)[:400000].astype(np.uint64) << np.uint64(20)) | t
    keys = np.concatenate([keys, (np.arange(100, dtype=np.uint64) << np.uint64(42)) | np.uint64(3 << 20)])
    g = engine.Lpma(V)
    g.update(ins=_dev(np.unique(keys)))
    k, v = g.export_sorted()
    srcs = rng.integers(0, V, n)
    srcs[[0, 5, n // 2, n - 1]] = 11
    wins = np.full(n, 0xFFFFF, np.uint64)
    wins[[5, n - 1]] = np.uint64(7 << 32 | 7)
    _check_lists(g, k, v, srcs, wins, V)
    g.close()


@pytest.mark.parametrize("V,case", [
    (1024, "even"), (1025, "even"), (5000, "even"), (40000, "even"),  # 1, 2, 5 and 40 bins
    (40000, "one"), (40000, "two"),  # every edge into one vertex, or into the last of a bin and the first of the next
])
def test_pagerank_by_destination(engine, oracle, V, case):
    rng = np.random.default_rng(V)
    n = 400000 if V > 2000 else 180000
    src = rng.integers(0, V - 7, n).astype(np.uint64)  # the last vertices have no out-edges
    if case == "even":
        dst = rng.integers(0, V, n).astype(np.uint64)
        dst[:100000] = rng.integers(2000 % V, 2000 % V + 40, 100000)  # one bin of several chunks
    else:
        dst = np.full(n, 3071, np.uint64) if case == "one" else np.where(rng.random(n) < 0.5, 3071, 3072).astype(np.uint64)
    # a pair may be there at several times
    keys = np.unique((src << np.uint64(42)) | (dst << np.uint64(20)) | rng.integers(0, 100000, n).astype(np.uint64))
    assert keys.size >= 1 << 17 and 24 * keys.size >= 3 << 20  # the form under test is the one that runs
    g = engine.Lpma(V)
    g.update(ins=_dev(keys))
    got = g.pagerank(0.85, 24).cpu().numpy()
    k, _ = g.export_sorted()
    # as test_gpu_reads: the sums' order is the only difference
    np.testing.assert_allclose(got, oracle.pagerank(k, V, 0.85, 24), rtol=1e-10, atol=0)
    g.close()


@pytest.mark.parametrize("V,n", [(1, 0), (31, 40), (96, 30), (97, 900), (200, 4000), (1500, 25000), (70000, 3000)])
def test_csr_view_tile_edges(engine, oracle, V, n):
    """Views of 1 to a few hundred tiles of 128 segments, whose starts fall on
    every remainder of the 16-byte stores."""
    from test_gpu_parity import assert_csr
    rng = np.random.default_rng(V)
    g, o = engine.Lpma(V), oracle.OracleLpma(V)
    for step in range(4):
        i = rng.permutation(V * V * 64)[:n + step].astype(np.uint64) if V < 1600 else rng.integers(0, 1 << 40, n + step).astype(np.uint64)
        keys = ((i % np.uint64(V)) << np.uint64(42)) | ((i // np.uint64(V) % np.uint64(V)) << np.uint64(20)) | \
            (i // np.uint64(V) // np.uint64(V) % np.uint64(1 << 20))
        keys = np.unique(keys)
        vals = rng.integers(1, 255, keys.size).astype(np.uint8)
        if keys.size:
            import torch
            g.update(ins=_dev(keys), ins_vals=torch.from_numpy(vals).cuda())
            o.update(ins=keys, ins_vals=vals)
        assert_csr(g, o)
    g.close()
