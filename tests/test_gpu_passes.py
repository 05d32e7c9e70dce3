"""The one-launch digit passes of the batch sort (tier multi_pass) and the
compaction behind it, against the oracle: batches around a tile and a chunk
group, digits that all keys share, and repeated keys, whose last value has to
win (the passes are stable)."""
import numpy as np
import pytest

from test_gpu_parity import _dev, _dev8, assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["spread", "rows", "repeats"])
@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 16385, 90000, 600001])
def test_multi_pass_batches(engine, oracle, n, kind):
    from lpma_gb300 import rpma
    V = 1 << 15
    rng = np.random.default_rng(n)
    src = rng.integers(0, V if kind == "spread" else 3, n).astype(np.uint64)
    dst = rng.integers(0, V if kind != "repeats" else max(2, n // 40), n).astype(np.uint64)
    keys = (src << np.uint64(42)) | ((dst % np.uint64(V)) << np.uint64(20))
    vals = rng.integers(0, 255, n).astype(np.uint8)
    g, o = engine.Lpma(V), oracle.OracleLpma(V)
    for b in range(21):
        rpma.tune_set(b, "multi_pass")
    try:
        g.update(ins=_dev(keys), ins_vals=_dev8(vals))
        o.update(ins=keys, ins_vals=vals)
        assert_same(g, o, "insert")
        gone = rng.permutation(keys)[: n // 2 + 1]
        g.update(dels=_dev(gone), ins=_dev(keys[:5]))
        o.update(dels=gone, ins=keys[:5])
        assert_same(g, o, "delete")
    finally:
        for b in range(21):
            rpma.tune_set(b, 0)
        g.close()
