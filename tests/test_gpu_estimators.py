"""The values of the equal-time estimators that ride on the wraps, where G is resident in one SM's shared
memory, in global memory (L = 13 .. 15, and small lattices beside them) and in a cluster's (L = 16), for
both forms of exp(-dt K) and both sweep modes: the oracle's means of every directional sweep.

Tolerances: a wrapped G drifts from a fresh one by the wrap error, some 1e-13 per slice at beta <= 1, and
the estimators average its entries, so 1e-10 per slice mean; the sums of the stored slices of the same
sweep agree to rounding (1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UP, DOWN = 0, 1


def _sums(G):
    N = G.shape[0]
    tr = np.trace(G)
    return np.array([2 - 2 * tr / N, ((1 - np.diag(G)) ** 2).sum() / N, (2 * (G * G).sum() - 2 * tr + N) / N])


def _check(hq, oracle, sizes, mode, sweep_mode=None):
    nt, pace = 7, 3
    cfg = [dict(nl=L, u=4.0, mu=-0.3, beta=0.7, nt=nt, stabilization_pace=pace, seed=20 + L, expk_mode=mode) for L in sizes]
    e = hq.Engine(cfg)
    if sweep_mode is not None:
        e.set_sweep_mode(sweep_mode)
    e.fields_random()
    e.init()
    os = []
    for L in sizes:
        o = oracle.OracleChain(L, u=4.0, mu=-0.3, beta=0.7, nt=nt, pace=pace, seed=20 + L)
        o.fields_random()
        o.init()
        os.append(o)
    for d in (UP, DOWN, UP, DOWN):
        e.reset_estimators()
        e.sweep(d, hq.SWEEP_MEASURE)
        est = e.estimators_all()
        for c, o in enumerate(os):
            o.sweep(d)
            assert np.array_equal(e.fields(c), o.fields()), (sizes[c], d)
            assert est[c, 3] == nt
            want = sum(_sums(o.g_slice(0, t)) for t in range(nt)) / nt
            assert np.abs(want - o.measure_equaltime()).max() <= 1e-12
            assert np.abs(est[c, :3] / nt - want).max() <= 1e-10, (sizes[c], d, est[c, :3] / nt - want)
    e.close()


@pytest.mark.parametrize("mode", [0, 1], ids=["dense", "separable"])
@pytest.mark.parametrize("L", [2, 3, 4, 7, 8, 9, 12, 13, 14, 15, 16])
def test_values_of_the_estimators(hq, oracle, L, mode):
    for sweep_mode in ((hq.SWEEP_LAUNCHES, hq.SWEEP_PERSISTENT) if L <= 12 else (None,)):
        _check(hq, oracle, [L], mode, sweep_mode)


def test_values_beside_a_chain_beyond_one_sm(hq, oracle):
    _check(hq, oracle, [3, 4, 9, 12, 13, 16], -1)


@pytest.mark.parametrize("L,mode", [(4, 0), (9, 0), (12, 0), (13, 0), (13, 1), (14, 1), (15, 1), (16, 0), (16, 1)])
def test_estimators_equal_the_stored_slices(hq, L, mode):
    nt = 12
    e = hq.Engine([dict(nl=L, u=3.0, mu=0.1, beta=1.2, nt=nt, stabilization_pace=5, seed=5, snapshots=1, expk_mode=mode)])
    e.fields_random()
    e.init()
    for d in (UP, DOWN):
        e.reset_estimators()
        e.sweep(d, hq.SWEEP_MEASURE | hq.SWEEP_SNAPSHOT)
        want = sum(_sums(e.g(0, hq.G_TT, t)) for t in range(nt))
        est = e.estimators(0)
        np.testing.assert_allclose(est[:3], want, rtol=1e-12)
        assert est[3] == nt
    e.close()
