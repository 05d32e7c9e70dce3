"""Whole-tree redistributions (root windows, rebuilds at another height) in
one pass, against the oracle: trees of few and many segments, updates spread
and crowded (a segment with hundreds, a run of segments with a dozen each),
deletes, expiry, and batches on both sides of the bulk-load rule."""
import numpy as np
import pytest

from test_gpu_front import DST, Three, _key

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,deg", [(40, 6), (300, 20), (1 << 12, 5), (1 << 12, 24), (1 << 15, 9)])
def test_spread_and_crowded(engine, oracle, V, deg):
    t = Three(engine, oracle, V)
    rng = np.random.default_rng(V + deg)
    half = V // 2  # vertices up to here hold the spread edges, dst above are for the crowds
    n = V * deg

    def spread(k, lo=0):
        return np.unique(_key(rng.integers(0, V, k), rng.integers(lo, max(lo + 1, half), k)))

    whole = 0
    t.update(ins=rng.permutation(spread(n)), where="load")
    hub = _key(np.full(V - half, V // 3), half + np.arange(V - half))          # one place, V / 2 keys
    run = np.unique(_key(np.repeat(np.arange(V // 4, V // 4 + V // 16 + 1), 9),   # a dozen a segment, a run of them
                         half + rng.integers(0, V - half, 9 * (V // 16 + 1))))
    steps = [("spread", spread(n // 3), None), ("run", run, None), ("hub", hub, None),
             ("spread again", spread(n // 2), 0.1), ("fewer", None, 0.75), ("hub gone", spread(n // 8), hub),
             ("fewer still", None, 0.8)]
    for name, ins, dels in steps:
        if isinstance(dels, float):
            dels = rng.permutation(t.live())[: int(dels * t.live().size)]
        vals = None if ins is None or name == "spread" else rng.integers(0, 255, ins.size).astype(np.uint8)
        order = None if ins is None else rng.permutation(ins.size)
        s = t.update(ins=None if ins is None else ins[order], vals=None if vals is None else vals[order], dels=dels, where=name)
        whole += s["root_executed"] or s["rebuilt"] or s["fill_empty"]
    assert whole >= 2
    t.close()


@pytest.mark.parametrize("V", [50, 1 << 12])
def test_with_expiry(engine, oracle, V):
    """Ticks of timestamped edges, all but the last few expired now and then."""
    t = Three(engine, oracle, V)
    rng = np.random.default_rng(V)
    whole = 0
    for tick in range(12):
        k = V * (9 if tick % 4 else 25)
        e = np.unique(_key(rng.integers(0, V, k), rng.integers(0, V, k)) >> DST) << DST
        hub = (_key(np.full(V // 2, V // 5), np.arange(V // 2)) >> DST) << DST
        e = np.union1d(e, hub) if tick % 3 == 0 else e
        s = t.update(ins=rng.permutation(e) | np.uint64(10 + tick), thres=(10 + tick - 2) if tick % 4 != 1 else 0,
                     where="tick %d" % tick)
        whole += s["root_executed"] or s["rebuilt"] or s["fill_empty"]
    assert whole >= 2
    t.close()


@pytest.mark.parametrize("share", [1.9, 2.1, 30.0])
def test_bulk_rule(engine, oracle, share):
    """share * segments keys into one tree: on both sides of the rule."""
    V = 1 << 11
    t = Three(engine, oracle, V)
    rng = np.random.default_rng(3)
    s = t.update(ins=np.unique(_key(rng.integers(0, V, 12000), rng.integers(0, V // 2, 12000))))
    nseg = (2 << s["height_after"]) - 1
    e = rng.permutation(np.unique(_key(rng.integers(0, V, 90000), rng.integers(V // 2, V, 90000))))
    t.update(ins=e[: int(share * nseg)], where="bulk")
    t.close()
