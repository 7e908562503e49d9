"""Every lattice size of the resident update path against the oracle: the edges of the 16-site
blocks (N = L*L from 1 to 144, odd and even, one block, a short last block), both forms of
exp(-dt K), the delay depths, ragged stabilisation intervals, and the first sizes that keep G in
global memory (L = 13) or in a cluster (L = 16).

Tolerances: the field trajectory is identical; a freshly stabilised G agrees to 1e-10 x max(1, |G|),
the bound of the other parity tests; the estimator sums average wrapped G's, whose drift per slice
is bounded by the wrap error, to 1e-9.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UP, DOWN = 0, 1


def _check(hq, oracle, L, nt, pace, mode, depth=0, u=4.0, mu=-0.3, sweep_mode=None, trips=2):
    cfg = dict(nl=L, u=u, mu=mu, beta=0.1 * nt, nt=nt, stabilization_pace=pace, expk_mode=mode, delay_depth=depth)
    e = hq.Engine([dict(cfg, seed=70 + L), dict(cfg, seed=71 + L)])
    if sweep_mode is not None:
        e.set_sweep_mode(sweep_mode)
    e.fields_random()
    e.init()
    for _ in range(trips):
        e.sweep(UP, hq.SWEEP_MEASURE)
        e.sweep(DOWN, hq.SWEEP_MEASURE)
    est = e.estimators_all()
    for c in range(2):
        o = oracle.OracleChain(L, nnt=1.0, u=u, mu=mu, beta=0.1 * nt, nt=nt, pace=pace, seed=70 + L + c)
        o.fields_random()
        o.init()
        for _ in range(trips):
            o.sweep(UP)
            o.sweep(DOWN)
        assert np.array_equal(e.fields(c), o.fields()), (L, c)
        g = o.g()
        assert np.abs(e.g(c) - g).max() <= 1e-10 * max(1.0, np.abs(g).max()), (L, c)
        assert est[c, 5] == o.counts()[1] and est[c, 3] == 2 * trips * nt
        assert np.isfinite(est[c]).all()
    e.close()


@pytest.mark.parametrize("L", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12])
def test_resident_sizes_separable(hq, oracle, L):
    _check(hq, oracle, L, nt=13, pace=5, mode=hq.EXPK_SEPARABLE)


@pytest.mark.parametrize("L", [2, 3, 4, 5, 7, 9, 12])
def test_resident_sizes_dense_persistent(hq, oracle, L):
    _check(hq, oracle, L, nt=8, pace=5, mode=hq.EXPK_DENSE, sweep_mode=hq.SWEEP_PERSISTENT)


@pytest.mark.parametrize("L,depth", [(4, 4), (5, 8), (6, 4), (9, 8), (12, 8)])
def test_delay_depths(hq, oracle, L, depth):
    _check(hq, oracle, L, nt=9, pace=4, mode=hq.EXPK_SEPARABLE, depth=depth)


@pytest.mark.parametrize("L", [13, 14, 16])
def test_sizes_beyond_one_sm(hq, oracle, L):
    _check(hq, oracle, L, nt=7, pace=4, mode=hq.EXPK_SEPARABLE, trips=1)


def test_small_lattices_beside_large_ones(hq, oracle):
    """A context whose largest chain does not fit one SM keeps every G in global memory."""
    cfg = [dict(nl=L, u=4.0, mu=0.0, beta=0.7, nt=7, stabilization_pace=4, seed=9 + L) for L in (3, 4, 8, 13)]
    e = hq.Engine(cfg)
    e.fields_random()
    e.init()
    e.sweep(UP, hq.SWEEP_MEASURE)
    e.sweep(DOWN, hq.SWEEP_MEASURE)
    for c, L in enumerate((3, 4, 8, 13)):
        o = oracle.OracleChain(L, nnt=1.0, u=4.0, mu=0.0, beta=0.7, nt=7, pace=4, seed=9 + L)
        o.fields_random()
        o.init()
        o.sweep(UP)
        o.sweep(DOWN)
        assert np.array_equal(e.fields(c), o.fields()), L
        assert np.abs(e.g(c) - o.g()).max() <= 1e-10, L
    e.close()


@pytest.mark.parametrize("L", [3, 8, 9, 12])
def test_measured_slices_equal_the_snapshots(hq, L):
    """The estimators that ride on the wraps equal those of the per-slice G's to rounding (1e-12)."""
    e = hq.Engine([dict(nl=L, u=3.0, mu=0.1, beta=1.2, nt=12, stabilization_pace=5, seed=5, snapshots=1)])
    e.fields_random()
    e.init()
    N = L * L
    for d in (UP, DOWN):
        e.reset_estimators()
        e.sweep(d, hq.SWEEP_MEASURE | hq.SWEEP_SNAPSHOT)
        est = e.estimators(0)
        want = np.zeros(3)
        for t in range(12):
            G = e.g(0, hq.G_TT, t)
            tr = np.trace(G)
            want += [2 - 2 * tr / N, ((1 - np.diag(G)) ** 2).sum() / N, (2 * (G * G).sum() - 2 * tr + N) / N]
        np.testing.assert_allclose(est[:3], want, rtol=1e-12)
        assert est[3] == 12
    e.close()
