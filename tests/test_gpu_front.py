"""The partitioned update front against the oracle and against the sorted
front, at the edges of what it does: the batch sizes where it starts and
where the bucket count changes, segments with more keys than a counter or a
window takes, keys that stop at (or at an empty one of) the top nodes,
buckets that overflow, and the stats, which must not tell the two apart."""
import numpy as np
import pytest

from test_gpu_parity import _dev, _dev8, assert_csr, assert_same

pytestmark = pytest.mark.gpu

STATS = ("height_before", "height_after", "n_ins_applied", "n_upserts", "n_del_applied", "n_noop", "root_executed",
         "eager_levelup", "overflow", "rebuilt", "levelup_path", "fill_empty", "levelup", "windows_single",
         "windows_small", "windows_big", "slots_rewritten", "slots_small", "num_items")
SRC, DST = np.uint64(42), np.uint64(20)


def _key(s, d, t=0):
    return (np.asarray(s, np.uint64) << SRC) | (np.asarray(d, np.uint64) << DST) | np.asarray(t, np.uint64)


class Three:
    """One graph on the partitioned front, one on the sorted front, one oracle."""

    def __init__(self, engine, oracle, V):
        from lpma_gb300 import rpma
        self.rpma = rpma
        self.g, self.h, self.o = engine.Lpma(V), engine.Lpma(V), oracle.OracleLpma(V)

    def update(self, ins=None, dels=None, vals=None, thres=0, where="", parted=None):
        d = dict(ins=None if ins is None else _dev(ins), dels=None if dels is None else _dev(dels),
                 ins_vals=None if vals is None else _dev8(vals), thres=thres)
        n = (0 if ins is None else ins.size) + (0 if dels is None else dels.size)
        b = max(0, int(n - 1).bit_length())
        sg = self.g.update(**d)
        self.rpma.tune_set(b, "tile_merge")
        try:
            sh = self.h.update(**d)
        finally:
            self.rpma.tune_set(b, 0)
        self.o.update(ins=ins, dels=dels, ins_vals=vals, thres=thres)
        assert_same(self.g, self.o, where)
        assert_same(self.h, self.o, where + " (sorted)")
        for k in STATS:
            assert sg[k] == sh[k], (where, k, sg[k], sh[k])
        if parted is not None:
            assert (sg["sort_passes"] == 1) == parted, (where, sg["sort_passes"])
        return sg

    def live(self):
        k, _ = self.o.export_sorted()
        return k[((k >> DST) & np.uint64(0x3FFFFF)) != np.uint64(0x3FFFFE)]

    def close(self):
        assert_csr(self.g, self.o)
        self.g.close()
        self.h.close()


@pytest.mark.parametrize("n", [255, 256, 257, 511, 1000, 4095, 4097, 30000])
def test_batches_of_n(engine, oracle, n):
    V = 1 << 13
    t = Three(engine, oracle, V)
    e = oracle.shuffle(oracle.rmat_edges(n, 13, 24), 3)
    t.update(ins=e[:60000], where="load")
    rng = np.random.default_rng(n)
    pos = 60000
    for step in range(4):
        live = t.live()
        ni = (n, 0, n - n // 3, n // 2)[step]
        ins = e[pos:pos + ni]
        pos += ni
        dels = rng.choice(live, n - ins.size, replace=False)
        if step == 3 and dels.size > 20:  # repeats, stored keys, absent deletes, keys on both sides
            ins = np.concatenate([ins, ins[:7], live[:9], dels[:3]])
            dels = np.concatenate([dels, dels[:5], e[-4:], ins[:2]])
        vals = rng.integers(0, 255, ins.size).astype(np.uint8) if step >= 2 and ins.size else None
        t.update(ins=ins if ins.size else None, dels=dels if dels.size else None, vals=vals,
                 where="n=%d step %d" % (n, step), parted=(n >= 256 or step == 3 and n > 240) if step < 3 else None)
    t.close()


@pytest.mark.parametrize("m", [30, 64, 65, 200, 256])
def test_many_keys_of_one_segment(engine, oracle, m):
    """m keys into one place of a large tree, among spread ones."""
    V = 1 << 13
    t = Three(engine, oracle, V)
    rng = np.random.default_rng(m)
    e = np.unique(_key(rng.integers(0, V, 90000), rng.integers(0, V // 2, 90000)))
    t.update(ins=e)
    spread = np.unique(_key(rng.integers(0, V, 3000), rng.integers(V // 2, V - 600, 3000)))
    close = _key(np.full(m, 4000), V - 500 + np.arange(m))
    batch = rng.permutation(np.concatenate([spread, close, close[: m // 2]]))
    t.update(ins=batch, where="insert", parted=True)
    t.update(dels=batch, where="delete", parted=True)
    t.close()


def test_keys_at_top_nodes_and_in_emptied_ranges(engine, oracle):
    """Vertices lose all their edges (segments empty out, some of them top
    nodes), then take edges again; batches of keys that lie between a top
    node's first and last key."""
    V = 1 << 12
    t = Three(engine, oracle, V)
    rng = np.random.default_rng(5)
    e = oracle.shuffle(oracle.rmat_edges(77, 12, 40), 3)
    t.update(ins=e)
    for step in range(6):
        live = t.live()
        lo = int(rng.integers(0, V - 700))
        src = (live >> SRC).astype(np.int64)
        gone = live[(src >= lo) & (src < lo + 600)]
        gone = gone[:20000]
        t.update(dels=gone, where="range %d gone" % step)
        back = rng.permutation(gone)[: gone.size // 2 + 300]
        if back.size:
            t.update(ins=back, where="range %d back" % step)
        k, _ = t.o.export_sorted()
        near = k[rng.integers(0, k.size, 2000)]
        near = near[((near >> DST) & np.uint64(0x3FFFFF)) < np.uint64(V - 2)] + (np.uint64(1) << DST)
        near = near[((near >> DST) & np.uint64(0x3FFFFF)) < np.uint64(V)]
        t.update(ins=np.unique(near), where="neighbours %d" % step)
    t.close()


def test_bucket_overflow_takes_the_sorted_front(engine, oracle):
    """5,000 keys of one vertex overflow their bucket: the batch is applied
    all the same, and so are the next ones, spread or not."""
    V = 1 << 14
    t = Three(engine, oracle, V)
    rng = np.random.default_rng(9)
    e = np.unique(_key(rng.integers(0, V, 200000), rng.integers(0, V // 2, 200000)))
    t.update(ins=e)
    crowd = rng.permutation(_key(np.full(5000, 77), V // 2 + np.arange(5000)))
    t.update(ins=crowd, where="crowd", parted=False)
    for step in range(18):
        spread = np.unique(_key(rng.integers(0, V, 1500), rng.integers(V // 2, V, 1500)))
        t.update(ins=spread, where="after %d" % step, parted=step >= 16)
    t.update(dels=crowd, where="crowd gone", parted=False)
    t.close()


def test_rejected_batch_changes_nothing(engine, oracle):
    from lpma_gb300 import LpmaError
    V = 1 << 12
    t = Three(engine, oracle, V)
    e = oracle.shuffle(oracle.rmat_edges(5, 12, 24), 3)
    t.update(ins=e[:40000])
    for bad in (_key([V], [0]), _key([0], [V]), np.array([2**64 - 1], np.uint64), _key([3], [0x3FFFFE])):
        ins = np.concatenate([e[40000:42000], bad])
        for kw in (dict(ins=_dev(ins)), dict(dels=_dev(ins))):
            with pytest.raises(LpmaError):
                t.g.update(**kw)
            assert_same(t.g, t.o, "rejected")
    with pytest.raises(LpmaError):
        t.g.update(ins=_dev(e[40000:42000]), thres=1)  # inserts older than the threshold
    assert_same(t.g, t.o, "rejected")
    t.update(ins=e[40000:42000], where="after", parted=True)
    t.close()


@pytest.mark.parametrize("batch", [300, 3000, 20000])
def test_expiry_thresholds(engine, oracle, batch):
    V = 1 << 12
    t = Three(engine, oracle, V)
    rng = np.random.default_rng(batch)
    for tick in range(1, 14):
        b = batch if tick > 6 else 9000
        keys = np.unique(_key(rng.integers(0, V, b), rng.integers(0, V, b), tick))
        dels = None
        if tick > 6:
            live = t.live()
            dels = rng.choice(live, min(b // 5, live.size), replace=False)  # some have expired
        t.update(ins=keys, dels=dels, thres=max(0, tick - 5), where="tick %d" % tick)
    t.close()


@pytest.mark.parametrize("batch", [100, 2000])
def test_expiry_of_equal_batches(engine, oracle, batch):
    """A threshold that moves with every call while the batch's shape stays
    (one captured front serves them all), with a rejected call in between."""
    from lpma_gb300 import LpmaError
    V = 1 << 11
    t = Three(engine, oracle, V)
    rng = np.random.default_rng(batch)
    edges = oracle.shuffle(oracle.rmat_edges(batch, 11, 24), 5)
    edges = np.unique((edges >> DST) << DST)
    edges = rng.permutation(edges)[: 14 * batch].reshape(14, batch)
    for tick in range(1, 29):
        ins = edges[tick % 14] | np.uint64(tick)
        s = t.update(ins=ins, thres=max(0, tick - 6), where="tick %d" % tick)
        assert s["n_ins_applied"] == batch
        if tick == 15:
            bad = np.append(ins[1:], _key([V], [0]))
            with pytest.raises(LpmaError):
                t.g.update(ins=_dev(bad), thres=tick - 6)
    t.close()
