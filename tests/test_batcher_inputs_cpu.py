"""What Batcher.update hands to the library, without a GPU: the library is a
stand-in that looks at the records it gets, the tensors are stand-ins whose
lifetime the test watches."""
import ctypes
import gc
import weakref

import pytest

from lpma_gb300 import _abi, rpma


class FakeTensor:
    """A contiguous device tensor of n keys at an address of its own."""
    dtype = "torch.int64"

    def __init__(self, address, n):
        self.address, self.n = address, n

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return self.address

    def numel(self):
        return self.n


class FakeGraph:
    def __init__(self, handle):
        self._h = ctypes.c_void_p(handle)


class FakeLib:
    """Notes the handles and records of lpma_update_batch, and which of the
    watched tensors are alive while the call runs."""

    def __init__(self, watched=()):
        self.watched = watched

    def lpma_update_batch(self, b, hs, items, n, stream, stats, status):
        gc.collect()
        self.alive = [r() is not None for r in self.watched]
        self.handles = [h or 0 for h in (ctypes.c_void_p * n).from_address(_address(hs))]
        self.items = [(x.ins, x.n_ins, x.dels, x.n_del, x.thres)
                      for x in (_abi.LpmaBatch * n).from_address(_address(items))]
        return 0


def _address(x):
    return x if isinstance(x, int) else ctypes.addressof(x)


@pytest.fixture
def batcher(monkeypatch):
    monkeypatch.setattr(rpma, "_stream_ptr", lambda stream: 0)
    b = rpma.Batcher.__new__(rpma.Batcher)
    b._b = None
    return b


def test_batches_of_an_iterator_live_until_the_call_returns(batcher):
    watched = []

    def batches():
        for i in range(6):
            t, d = FakeTensor(0x1000 * (i + 1), 10 + i), FakeTensor(0x100000 * (i + 1), 3)
            watched.extend((weakref.ref(t), weakref.ref(d)))
            yield {"ins": t, "dels": d} if i % 2 else (t, d)
            del t, d

    batcher._L = FakeLib(watched)
    batcher.update([FakeGraph(0x10 * (i + 1)) for i in range(6)], batches())
    assert batcher._L.alive == [True] * 12
    assert batcher._L.items == [(0x1000 * (i + 1), 10 + i, 0x100000 * (i + 1), 3, 0) for i in range(6)]
    gc.collect()
    assert all(r() is None for r in watched)  # and no longer


@pytest.mark.parametrize("n_batches", [0, 2, 3, 4])
def test_graphs_without_a_batch_get_no_handle(batcher, n_batches):
    """The library refuses a null handle (invalid argument), so a call with
    fewer batches than graphs is refused for the graphs left over; batches
    beyond the graphs are not looked at."""
    batcher._L = FakeLib()
    graphs = [FakeGraph(0x10 * (i + 1)) for i in range(3)]
    batches = [(FakeTensor(0x1000 * (i + 1), i + 1), None) for i in range(n_batches)]
    batcher.update(graphs, batches)
    m = min(n_batches, 3)
    assert batcher._L.handles == [0x10 * (i + 1) for i in range(m)] + [0] * (3 - m)
    assert batcher._L.items == [(0x1000 * (i + 1), i + 1, None, 0, 0) for i in range(m)] + [(None, 0, None, 0, 0)] * (3 - m)
