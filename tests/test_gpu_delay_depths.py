"""Delay depths 4 and 8, whose blocks have walks of their own, where G is beyond one SM's shared memory,
and last blocks of 4 sites (N = 36, 100) and of one (N = 49) at depths 16 and 8: the oracle's field trajectory, and G to 1e-10 x max(1, |G|), the bound of the other
parity tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UP, DOWN = 0, 1


@pytest.mark.parametrize("log", [False, True], ids=["", "ratio_log"])
@pytest.mark.parametrize("L,depth", [(13, 4), (13, 8), (14, 4), (16, 4), (16, 8), (6, 16), (10, 16), (10, 8), (7, 8)])
def test_walks_of_short_blocks(hq, oracle, L, depth, log):
    nt, pace = 6, 4
    e = hq.Engine([dict(nl=L, u=4.0, mu=-0.2, beta=0.6, nt=nt, stabilization_pace=pace, seed=90 + L, delay_depth=depth)])
    assert e.config(0)[1] == depth
    o = oracle.OracleChain(L, nnt=1.0, u=4.0, mu=-0.2, beta=0.6, nt=nt, pace=pace, seed=90 + L)
    e.fields_random(0)
    o.fields_random()
    e.init()
    o.init()
    if log:
        e.ratio_log(0, capacity=2 * nt * L * L)
    for d in (UP, DOWN):
        e.sweep(d, hq.SWEEP_MEASURE | (hq.SWEEP_LOG_RATIOS if log else 0))
        o.sweep(d)
        assert np.array_equal(e.fields(0), o.fields())
        assert np.abs(e.g(0) - o.g()).max() <= 1e-10 * max(1.0, np.abs(o.g()).max())
    assert e.estimators(0)[5] == o.counts()[1]
    if log:
        assert len(e.ratio_log(0)) == 2 * nt * L * L
    e.close()
