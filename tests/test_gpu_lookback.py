"""The digit passes of the batch sort whose tiles do not hear of one another.

A tile waits, with a bound, for the counts that the tiles before it publish.
When a wait runs out, the tile counts the digits of the keys before it itself.
The test setting (lpma_debug_sort_barrier) lets a wait run out after one poll,
or takes none of the published words.  Every sort is right all the same: the
callers that cannot report an error (the fixed-scratch shuffle is asynchronous)
depend on that.  Nothing hangs or faults: the waits run out by design, and the
counting reads the pass's input only."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import _dev, _dev8, assert_same

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1], ids=["one_poll", "deaf"])
def deaf(engine, request):
    import torch
    from lpma_gb300 import _abi
    L = _abi.load()
    torch.cuda.synchronize()
    _abi.check(L.lpma_debug_sort_barrier(1, request.param), "lpma_debug_sort_barrier")
    yield L
    torch.cuda.synchronize()
    L.lpma_debug_sort_barrier(0, 0)


@pytest.mark.parametrize("n", [4096, 4097, 20000, 65536])
def test_shuffles(engine, oracle, deaf, n):
    import torch
    from lpma_gb300 import _abi
    keys = np.random.default_rng(n).integers(0, 1 << 62, n).astype(np.uint64)
    want = oracle.shuffle(np.sort(keys), 9)
    a, b = _dev(keys), _dev(keys)
    engine.shuffle_device(9, a)
    _abi.check(deaf.lpma_shuffle_static(9, ctypes.c_void_p(b.data_ptr()), n, None), "lpma_shuffle_static")
    torch.cuda.synchronize()
    assert np.array_equal(a.cpu().numpy().view(np.uint64), want)
    assert np.array_equal(b.cpu().numpy().view(np.uint64), want)


def test_generator(engine, oracle, deaf):
    import torch
    out = torch.empty(16 << 16, dtype=torch.int64, device="cuda")
    n = engine.gen_rmat_device(11, 16, 16, out)
    assert np.array_equal(out[:n].cpu().numpy().view(np.uint64), oracle.rmat_edges(11, 16, 16))


def test_update_keeps_the_order_of_equal_keys(engine, oracle, deaf):
    from lpma_gb300 import rpma
    V, n = 1 << 12, 30000
    rng = np.random.default_rng(3)
    keys = (rng.integers(0, V, n).astype(np.uint64) << np.uint64(42)) | (rng.integers(0, 20, n).astype(np.uint64) << np.uint64(20))
    vals = rng.integers(0, 255, n).astype(np.uint8)
    g, o = engine.Lpma(V), oracle.OracleLpma(V)
    rpma.tune_set(int(n - 1).bit_length(), "multi_pass")
    try:
        g.update(ins=_dev(keys), ins_vals=_dev8(vals))
    finally:
        rpma.tune_set(int(n - 1).bit_length(), 0)
    o.update(ins=keys, ins_vals=vals)
    assert_same(g, o, "insert")
    g.close()
