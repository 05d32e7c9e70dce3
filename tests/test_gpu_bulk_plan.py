"""A bulk load whose items fit a tree of one more level exactly, or not by
one key: the planner plans windows in the first case and none in the second
(a rebuild from the whole list)."""
import numpy as np
import pytest

from test_gpu_parity import _dev, assert_csr, assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [5, 64, 700])
@pytest.mark.parametrize("over", [-1, 0, 1, 2])
def test_bulk_load_at_the_next_levels_capacity(engine, oracle, V, over):
    g, o = engine.Lpma(V), oracle.OracleLpma(V)
    slots = 32 * ((2 << (g.height + 1)) - 1)  # of a tree one level higher
    n = slots + over - V
    rng = np.random.default_rng(V + over)
    i = rng.permutation(V * V * 64)[:n].astype(np.uint64)  # (src, dst, t)
    keys = ((i % np.uint64(V)) << np.uint64(42)) | ((i // np.uint64(V) % np.uint64(V)) << np.uint64(20)) | \
        (i // np.uint64(V * V))
    sg, so = g.update(ins=_dev(keys)), o.update(ins=keys)
    assert g.num_items == slots + over
    for k in ("overflow", "levelup", "levelup_path", "rebuilt"):
        assert sg[k] == so[k], k
    assert_same(g, o, "V=%d over=%d" % (V, over))
    assert_csr(g, o)
    g.close()
