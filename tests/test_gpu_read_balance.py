"""Read paths whose work is split by segments, at the edges of the split:
hubs whose slots fill a few segments more or less than one range of the BFS
frontier (4 segments of 32 slots), vertices without edges, every source the
same."""
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
