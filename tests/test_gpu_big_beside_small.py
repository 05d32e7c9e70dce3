"""Big windows (more than 32 segments) that execute in one loop with small
ones: the counts of the small windows' segments hold their updates already,
so the big windows' places in the gathered copy must not depend on them."""
import pytest

from test_gpu_parity import _dev, assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,ef,seed,frac", [(13, 16, 40, 0.5), (13, 16, 569, 0.6), (11, 18, 55, 0.6), (11, 18, 70, 0.6),
                                                (12, 14, 3, 0.5)])
def test_half_into_half(engine, oracle, scale, ef, seed, frac):
    V = 1 << scale
    e = oracle.shuffle(oracle.rmat_edges(seed, scale, ef), seed)
    half = int(e.size * (1 - frac))
    g, o = engine.Lpma(V), oracle.OracleLpma(V)
    for part in (e[:half], e[half:]):
        g.update(ins=_dev(part))
        o.update(ins=part)
        assert_same(g, o, "insert")
    for part in (e[:half], e[half:]):
        g.update(dels=_dev(part))
        o.update(dels=part)
        assert_same(g, o, "delete")
    g.close()
