"""The partitioned front's buckets on tall trees: few buckets for a batch of
some hundred keys, so a bucket's subtree is higher than the levels staged in
shared memory (the descent goes on in global memory) and one counter stands for
several segments (which decides where the warps cut their shares)."""
import numpy as np
import pytest

from test_gpu_parity import _dev, _dev8, assert_same

pytestmark = pytest.mark.gpu

V = 1 << 16


def _key(src, dst):
    return (np.asarray(src).astype(np.uint64) << np.uint64(42)) | (np.asarray(dst).astype(np.uint64) << np.uint64(20))


@pytest.fixture(scope="module")
def tall(engine, oracle):
    rng = np.random.default_rng(15)
    base = np.unique(_key(rng.integers(0, V, 2200000), rng.integers(0, V, 2200000)))
    g, o = engine.Lpma(V), oracle.OracleLpma(V)
    g.update(ins=_dev(base))
    o.update(ins=base)
    # 2^3 to 2^5 buckets for the batches below: subtrees of height 11 to 13
    assert o.height >= 16
    yield g, o, base
    g.close()


def _batches(rng, n, kind, base):
    """(inserts, deletes), n keys together."""
    if kind == "spread":
        src, dst = rng.integers(0, V, n), rng.integers(0, V, n)
    elif kind == "crowded":  # a few neighbouring vertices: far more than 64 keys a counter
        src, dst = rng.integers(777, 780, n), rng.integers(0, V, n)
        # (1,024 of them at most fit one bucket)
    else:  # places of about ten keys each, here and there
        src = np.repeat(rng.integers(0, V, n // 10 + 1), 10)[:n]
        dst = rng.integers(0, 500, n)
    keys = _key(src, dst)
    stored = base[rng.integers(0, base.size, n)]
    if kind == "crowded":
        a = np.searchsorted(base, _key(777, 0))
        stored = base[a + rng.integers(0, 60, n)]
    ins = np.concatenate([keys[: n // 2], keys[: n // 8], stored[: n // 8]])          # repeats, upserts
    dels = np.concatenate([stored[n // 8: n // 4], keys[: n // 16], keys[n // 2:]])    # stored, just inserted, absent
    return rng.permutation(ins), rng.permutation(dels)


@pytest.mark.parametrize("kind", ["spread", "crowded", "places"])
@pytest.mark.parametrize("n", [256, 600, 1000])
def test_few_keys_on_a_tall_tree(tall, n, kind):
    g, o, base = tall
    if kind == "crowded":
        n = min(n, 700)
    rng = np.random.default_rng(n)
    for turn in range(3):
        ins, dels = _batches(rng, n, kind, base)
        vals = rng.integers(0, 255, ins.size).astype(np.uint8)
        sg = g.update(ins=_dev(ins), ins_vals=_dev8(vals), dels=_dev(dels))
        so = o.update(ins=ins, ins_vals=vals, dels=dels)
        assert sg["sort_passes"] == 1  # the partitioned front took it
        for k in ("n_ins_applied", "n_del_applied", "n_upserts", "n_noop", "root_executed", "overflow"):
            assert sg[k] == so[k], (k, turn)
        assert_same(g, o, "turn %d" % turn)
    assert g.height == o.height >= 16


@pytest.mark.parametrize("kind", ["spread", "crowded"])
def test_ticks_on_a_tall_tree(engine, oracle, kind):
    """The same with an expiry threshold."""
    rng = np.random.default_rng(3)
    base = np.unique(_key(rng.integers(0, V, 2200000), rng.integers(0, V, 2200000))) | np.uint64(5)
    base[::50] -= np.uint64(4)  # these expire
    g, o = engine.Lpma(V), oracle.OracleLpma(V)
    g.update(ins=_dev(base))
    o.update(ins=base)
    for t in (6, 7):
        ins, dels = _batches(rng, 700, kind, base)
        ins = (ins & ~np.uint64(0xFFFFF)) | np.uint64(t)
        sg = g.update(ins=_dev(ins), dels=_dev(dels), thres=t - 4)
        o.update(ins=ins, dels=dels, thres=t - 4)
        assert sg["sort_passes"] == 1
        assert_same(g, o, "tick %d" % t)
    g.close()
