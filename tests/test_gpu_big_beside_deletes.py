"""One call whose small windows lose keys and whose big window (more than 32
segments, not the root) gains some, further right.

The big windows' prefixes are taken after the small windows of the same call
have executed: the counts then hold a small window's result while the list
still has its deletes, so a segment that was spread full again counts fewer
items than the list deletes from it.  The start of the big window's updates in
the list must not depend on that."""
import numpy as np
import pytest

from test_gpu_parity import _dev, _dev8, assert_csr, assert_same

pytestmark = pytest.mark.gpu

KEY_NONE = np.uint64((1 << 64) - 1)


def _key(src, dst):
    return (np.uint64(src) << np.uint64(42)) | (np.asarray(dst, dtype=np.uint64) << np.uint64(20))


def _segments(o, keys):
    """Linear segment that each key is located in."""
    return o.locate(keys).astype(np.int64) // 32


def _counts(o):
    """Keys of each linear segment."""
    k, _ = o.layout()
    n = (k.reshape(-1, 32) != KEY_NONE).sum(axis=1)  # in the slots' order
    j = np.arange(1, n.size + 1)
    level = np.array([int(x).bit_length() - 1 for x in j])
    linear = ((2 * (j - (1 << level)) + 1) << (o.height - level)) - 1
    cnt = np.empty(n.size, np.int64)
    cnt[linear] = n
    return cnt


def scenario(oracle, scale, every, keep, n_big):
    """A graph of 2^scale vertices with 24 edges each, and a batch: of every
    `every`-th segment in the left half all stored edges but `keep` go, and
    n_big edges come to one vertex near the right end."""
    V = 1 << scale
    rng = np.random.default_rng(scale * 1000 + every)
    base = np.concatenate([_key(s, rng.choice(V, 24, replace=False)) for s in range(V)])
    vals = rng.integers(1, 255, base.size).astype(np.uint8)
    o = oracle.OracleLpma(V, skip_rule=False)
    o.update(ins=base, ins_vals=vals)
    seg = _segments(o, base)
    nseg = (2 << o.height) - 1
    go = []
    for s in range(3, nseg // 2, every):
        go.append(base[seg == s][keep:])
    dels = rng.permutation(np.concatenate(go))
    hub = V - 3
    new = np.setdiff1d(np.arange(V, dtype=np.uint64), (base[base >> np.uint64(42) == hub] >> np.uint64(20)) & np.uint64(0x3FFFFF))
    ins = _key(hub, rng.permutation(new)[:n_big])
    ins_vals = rng.integers(1, 255, ins.size).astype(np.uint8)
    return V, o, base, vals, ins, ins_vals, dels


def check_shape(o, ins, dels):
    """The oracle's update has the windows that the test is about: several
    segments end up with fewer keys than the batch deletes from them, left of a
    big window that is not the root."""
    nseg = (2 << o.height) - 1
    d = np.bincount(_segments(o, dels), minlength=nseg)
    i = np.bincount(_segments(o, ins), minlength=nseg)
    H = o.height
    st = o.update(ins=ins, dels=dels)
    assert o.height == H and not st["root_executed"] and not st["overflow"]
    assert sum(st["win_count"][6:H + 1]) == 1 and sum(st["win_count"][1:6]) > 0
    short = np.nonzero(_counts(o) - d + i < 0)[0]
    assert short.size >= 3 and short.max() < np.nonzero(i)[0].min()


@pytest.mark.parametrize("tier", [None, "tile_merge"])  # the partitioned front, the sorted front
@pytest.mark.parametrize("scale,every,keep,n_big", [(11, 7, 2, 700), (12, 40, 1, 1000), (12, 9, 3, 500)])
def test_deletes_left_of_a_big_window(engine, oracle, scale, every, keep, n_big, tier):
    from lpma_gb300 import rpma
    V, probe, base, vals, ins, ins_vals, dels = scenario(oracle, scale, every, keep, n_big)
    check_shape(probe, ins, dels)
    cfg = rpma.default_config()
    cfg.skip_rule = 0  # every level's windows
    o, g = oracle.OracleLpma(V, skip_rule=False), engine.Lpma(V, config=cfg)
    o.update(ins=base, ins_vals=vals)
    g.update(ins=_dev(base), ins_vals=_dev8(vals))
    assert_same(g, o, "loaded")
    bucket = int(ins.size + dels.size - 1).bit_length()
    if tier:
        rpma.tune_set(bucket, tier)
    try:
        sg = g.update(ins=_dev(ins), ins_vals=_dev8(ins_vals), dels=_dev(dels))
    finally:
        rpma.tune_set(bucket, 0)
    so = o.update(ins=ins, ins_vals=ins_vals, dels=dels)
    assert sg["windows_big"] == 1 and (sg["sort_passes"] == 1) == (tier is None)
    for k in ("n_ins_applied", "n_del_applied", "n_upserts", "n_noop"):
        assert sg[k] == so[k], k
    assert_same(g, o, "mixed")
    assert_csr(g, o)
    g.close()
