"""The edges of the kernels' size rules against the oracle: the one-launch equal-time G at every
lattice size it takes, the products and the factorisation's register panels beyond one SM's shared
memory, the displaced estimators at odd sizes, and the default sweep mode on both sides of its line.

Tolerances: a freshly stabilised G, the displaced G's and the estimators made of them agree to
1e-10 x max(1, |value|), the bound of the other parity tests; field trajectories are identical.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UP, DOWN, DYN = 0, 1, 2


def _close(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return np.abs(a - b).max() <= 1e-10 * max(1.0, np.abs(b).max())


# one stack entry, a ragged last interval, a pace of one, the sixteen entries that are allowed
@pytest.mark.parametrize("nt,pace", [(6, 6), (13, 5), (16, 1), (47, 3)])
@pytest.mark.parametrize("L", [1, 2, 3, 4, 5, 6, 7, 8])
def test_one_launch_equaltime_g(hq, oracle, L, nt, pace):
    import torch
    N = L * L
    o = oracle.OracleChain(L, nnt=1.0, u=4.0, mu=-0.3, beta=0.1 * nt, nt=nt, pace=pace, seed=30 + L)
    o.fields_random()
    o.init()
    f = torch.tensor(o.fields().astype(np.int8), device="cuda")
    g = torch.full((N + 1, N), float("nan"), dtype=torch.float64, device="cuda")  # a row behind, to stay as it is
    rc = hq.lib().hq_equaltime_g_noalloc(L, 1.0, 4.0, -0.3, 0.1 * nt, nt, pace, f.data_ptr(), g.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream)
    assert rc == 0, hq.capi.last_error()
    g = g.cpu().numpy()
    assert np.isnan(g[N]).all()
    assert _close(g[:N].T, o.g())


@pytest.mark.parametrize("mode", [0, 1], ids=["dense", "separable"])
@pytest.mark.parametrize("L,dynamic", [(3, True), (5, True), (7, True), (9, True), (13, True), (15, False), (16, False)])
def test_builders_and_panels(hq, oracle, L, dynamic, mode):
    nt, pace = (7, 3) if L < 13 else (5, 2)
    e = hq.Engine([dict(nl=L, u=4.0, mu=0.2, beta=0.1 * nt, nt=nt, stabilization_pace=pace, seed=5, expk_mode=mode,
                        dynamic=int(dynamic), snapshots=int(dynamic))])
    o = oracle.OracleChain(L, u=4.0, mu=0.2, beta=0.1 * nt, nt=nt, pace=pace, equaltime=True, dynamic=dynamic, seed=5)
    e.fields_random(0)
    o.fields_random()
    e.init()
    o.init()
    for d in (UP, DOWN):
        e.sweep(d)
        o.sweep(d)
    assert np.array_equal(e.fields(0), o.fields())
    assert _close(e.g(0), o.g())
    if dynamic:
        e.sweep(DYN)
        o.sweep(DYN)
        for which, idx in ((hq.G_TT, 0), (hq.G_T0, 1), (hq.G_0T, 2)):
            for t in range(nt):
                assert _close(e.g(0, which, t), o.g_slice(idx, t)), (which, t)
        sp, ld, _ = e.dynamic_estimators(0)
        osp, old, _ = o.measure_dynamic([0])
        assert _close(sp, osp) and _close(ld, old)
    e.close()


@pytest.mark.parametrize("L,n,persistent", [(6, 1, True), (6, 200, True), (7, 2, True), (8, 148, True), (7, 149, False),
                                            (9, 1, False)])
def test_default_sweep_mode(hq, L, n, persistent, monkeypatch):
    """Chains of up to 36 sites run persistently, those of up to 64 while there are no more than SMs (148);
    the other mode gives the same fields and, within the bound above, the same G."""
    monkeypatch.delenv("HQ_SWEEP_MODE", raising=False)
    cfg = [dict(nl=L, u=4.0, mu=0.1, beta=0.6, nt=6, stabilization_pace=4, seed=50 + c) for c in range(n)]
    a, b = hq.Engine(cfg), hq.Engine(cfg)
    assert a.sweep_mode() == (hq.SWEEP_PERSISTENT if persistent else hq.SWEEP_LAUNCHES)
    b.set_sweep_mode(hq.SWEEP_LAUNCHES if persistent else hq.SWEEP_PERSISTENT)
    for e in (a, b):
        e.fields_random()
        e.init()
        e.sweep(UP, hq.SWEEP_MEASURE)
        e.sweep(DOWN, hq.SWEEP_MEASURE)
    for c in (0, n // 2, n - 1):
        assert np.array_equal(a.fields(c), b.fields(c)), c
        assert _close(a.g(c), b.g(c)), c
    a.close()
    b.close()
