"""The partitioned front of the flat (GPMA) array against the oracle, at the
edges of what it does: the batch sizes where it starts and where the bucket
count changes, repeated keys and keys on both sides, crowded segments,
buckets that overflow, arrays whose segments have 8 and 16 slots, emptied
ranges, and rejected batches."""
import numpy as np
import pytest

from test_gpu_gpma import assert_same, gkeys, make
from test_gpu_parity import _dev, _dev8

pytestmark = pytest.mark.gpu

STATS = ("n_ins_applied", "n_upserts", "n_del_applied", "n_noop", "rebuilt", "overflow", "root_executed")


def both(g, o, where, ins=None, vals=None, dels=None):
    sg = g.update(ins=None if ins is None else _dev(ins), ins_vals=None if vals is None else _dev8(vals),
                  dels=None if dels is None else _dev(dels))
    so = o.update(ins=ins, ins_vals=vals, dels=dels)
    for k in STATS:
        assert sg[k] == so[k], (where, k, sg[k], so[k])
    assert_same(g, o, where)


@pytest.mark.parametrize("scale,n", [(9, 1), (9, 2), (9, 127), (9, 128), (12, 257), (12, 1000), (13, 4095), (13, 4097), (14, 40000),
                                     (17, 300000), (17, 700000)])
def test_batches_of_n(engine, oracle, scale, n):
    V = 1 << scale
    e = gkeys(oracle.shuffle(oracle.rmat_edges(n, scale, 16), 3))
    half = min(e.size // 2, 400000)
    g, o = make(engine, oracle, V)
    both(g, o, "load", ins=e[:half])
    rng = np.random.default_rng(n)
    pos = half
    for step in range(4):
        ni = (n, 0, n - n // 3, n // 2)[step]
        ins = e[pos:pos + ni]
        pos += ni
        dels = rng.choice(e[:pos], n - ins.size, replace=False)
        if step == 3:  # repeats, stored keys, absent and tombstoned deletes, keys on both sides
            ins = np.concatenate([ins, ins[:7], e[:9], dels[:3], ins[2:5]])
            dels = np.concatenate([dels, dels[:5], e[-4:], ins[:2]])
        vals = rng.integers(0, 255, ins.size).astype(np.uint8) if step >= 2 else None
        both(g, o, "n=%d step %d" % (n, step), ins=ins if ins.size else None, vals=vals,
             dels=dels if dels.size else None)
    g.close()


def test_crowds_overflow_and_emptied_ranges(engine, oracle):
    V = 1 << 13
    rng = np.random.default_rng(4)
    e = gkeys(oracle.shuffle(oracle.rmat_edges(8, 13, 16), 3))
    g, o = make(engine, oracle, V)
    both(g, o, "load", ins=e[:60000])
    spread = e[60000:90000]
    for m, k in ((300, 3000), (1025, 5000), (3000, 9000), (0, 700)):
        # m keys of one vertex among k spread ones: in one bucket, in some
        # of these batches more than it holds
        crowd = (np.uint64(777) << np.uint64(32)) | (np.arange(m, dtype=np.uint64) + np.uint64(4000))
        batch = rng.permutation(np.concatenate([crowd, spread[:k]]))
        both(g, o, "crowd %d" % m, ins=batch)
        both(g, o, "crowd %d gone" % m, dels=batch)
    for step in range(18):  # past the batches that the sorted front takes after an overflow
        both(g, o, "spread %d" % step, ins=spread[step * 1500:(step + 1) * 1500])
    low = e[:90000][(e[:90000] >> np.uint64(32)) < V // 2]
    both(g, o, "half empty", dels=low)
    both(g, o, "rewritten", ins=e[90000:100000])
    both(g, o, "back", ins=low[:20000], dels=spread[:2000])
    g.close()


def test_rejected_batch_changes_nothing(engine, oracle):
    from lpma_gb300 import LpmaError
    V = 1 << 11
    e = gkeys(oracle.shuffle(oracle.rmat_edges(6, 11, 16), 3))
    g, o = make(engine, oracle, V)
    both(g, o, "load", ins=e[:9000])
    for bad in (np.uint64(V) << np.uint64(32), np.uint64(V), np.uint64(2**64 - 1)):
        keys = np.append(e[9000:10000], bad)
        for kw in (dict(ins=_dev(keys)), dict(dels=_dev(keys))):
            with pytest.raises(LpmaError):
                g.update(**kw)
            assert_same(g, o, "rejected")
    with pytest.raises(LpmaError):
        g.update(ins=_dev(e[9000:10000]), ins_vals=_dev8(np.full(1000, 255, np.uint8)))
    assert_same(g, o, "rejected value")
    both(g, o, "after", ins=e[9000:10000])
    g.close()
